// Check of the rule by which kernels access host arrays directly
// (csrc/host_view.h).  Without arguments: the rule on made-up ranges.  With
// "gpu": what the driver reports of real allocations and registrations, in the
// main thread and as the first call of another; no kernel runs.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>

#include "host_view.h"

using namespace owt;

static int bad = 0;
static void expect(const char *what, bool got, bool want) {
  if (got != want) {
    ++bad;
    std::printf("%s: %s, want %s\n", what, got ? "direct" : "staged", want ? "direct" : "staged");
  }
}

static void rule() {
  HostRange r;
  r.pinned = r.readable = r.writable = true;
  r.start = 0x10000;
  r.size = 4096;
  r.device = 0x10000;
  auto ok = [&](uintptr_t p, size_t n, bool write = true) {
    HostRange q = r;
    q.device = p + (r.device - r.start);
    return host_view(q, p, n, write) == reinterpret_cast<void *>(q.device);
  };
  expect("the whole range", ok(0x10000, 4096), true);
  expect("its end", ok(0x10ff0, 16), true);
  expect("one value beyond its end", ok(0x10000, 4112), false);
  expect("starting inside, ending beyond", ok(0x10ff0, 32), false);
  expect("starting before it", ok(0xfff0, 32), false);
  expect("beyond it", ok(0x11010, 16), false);
  expect("a size that wraps around", ok(0x10010, SIZE_MAX - 8), false);
  expect("an address of 8 bytes' alignment", ok(0x10008, 16), false);
  r.writable = false;
  expect("a read of a read-only range", ok(0x10000, 4096, false), true);
  expect("a write to a read-only range", ok(0x10000, 4096, true), false);
  r.readable = false;
  expect("a range out of the GPU's reach", ok(0x10000, 4096, false), false);
  r.readable = r.writable = true;
  r.device = 0x50000;
  expect("another device address", ok(0x10100, 256), true);
  r.pinned = false;
  expect("pageable memory", ok(0x10000, 4096), false);
}

static bool direct(const void *p, size_t n, bool write = true) {
  return host_view(host_range(p), reinterpret_cast<uintptr_t>(p), n, write) != nullptr;
}

static void real() {
  constexpr size_t P = 1 << 16, N = 1 << 20;  // pages of at most 64 KiB
  char *a = nullptr;
  if (cudaHostAlloc(reinterpret_cast<void **>(&a), N, cudaHostAllocDefault) != cudaSuccess) std::exit(2);
  bool other = false;
  std::thread([&] { other = direct(a, N); }).join();
  expect("a page-locked array, from a new thread", other, true);
  expect("a page-locked array", direct(a, N), true);
  expect("its second half", direct(a + N / 2, N / 2), true);
  expect("more than it holds", direct(a, N + 16), false);
  char *m = static_cast<char *>(std::aligned_alloc(P, 8 * P));
  std::memset(m, 0, 8 * P);
  expect("a pageable array", direct(m, P), false);
  // pages 0, 1 and 3 registered, 2 not
  if (cudaHostRegister(m, 2 * P, cudaHostRegisterDefault) != cudaSuccess) std::exit(3);
  if (cudaHostRegister(m + 3 * P, P, cudaHostRegisterDefault) != cudaSuccess) std::exit(4);
  expect("a registered part", direct(m, 2 * P), true);
  expect("an array registered in part", direct(m, 3 * P), false);
  expect("an array with a hole, both ends registered", direct(m, 4 * P), false);
  if (cudaHostRegister(m + 2 * P, P, cudaHostRegisterDefault) != cudaSuccess) std::exit(5);
  expect("an array registered in three pieces", direct(m, 4 * P), false);
  void *d = nullptr, *u = nullptr;
  if (cudaMalloc(&d, 4096) != cudaSuccess || cudaMallocManaged(&u, 4096) != cudaSuccess) std::exit(6);
  expect("device memory", direct(d, 4096), false);
  expect("managed memory", direct(u, 4096), false);
  for (int b : {0, 2, 3}) cudaHostUnregister(m + b * P);
  expect("an array no longer registered", direct(m, P), false);
  cudaFree(d);
  cudaFree(u);
  cudaFreeHost(a);
  std::free(m);
}

int main(int argc, char **argv) {
  if (argc > 1 && !std::strcmp(argv[1], "gpu")) real();
  else rule();
  return bad ? 1 : 0;
}
