// DY1 along y for caller-owned device arrays, without any device allocation.
//
// Some callers cannot call cudaMalloc: programs that hand the whole device
// memory to their own pool allocator and forbid allocations from elsewhere,
// and tight loops that cannot accept the implicit device-wide
// synchronisation cudaMalloc and cudaFree bring.  owt_dy1_noalloc serves
// them: it needs no handle (creating one allocates) and keeps everything in
// the shared memory of its blocks.
//
// What it computes is the handle-based DY1 (owt_dy_apply with order 1):
// out = diag(c11) A1^-1 B1 in along y, for every line, with the compact first
// derivative of src/compdiff.hpp:11-69 and c11 = 1/(dy/ds) of
// src/solver.cpp:77,94 on the grid y = tanh(alpha s)/tanh(alpha).
//
// One launch.  Each block builds the tables for (NY, alpha) itself
// (noalloc_setup.h) and takes a tile of lines, all NY rows of which stay in
// shared memory: B1 on the way in, the band solve in place, c11 on the way
// out.  Bound by FP64 issue: a line component costs five FP64 operations a
// row in the solve, which is sequential in y, and five in the two parallel
// phases around it.  A tile is ceil(lines / SMs) lines, so that every SM
// works on one, at most 64 (one thread per component) and what fits beside
// the tables.  129 rows x 4096 lines: 633 us with one thread building the
// tables in a kernel of its own and a scratch array in device memory, 106 us
// now (the same bits).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>
#include <string>

#include "noalloc_setup.h"
#include "owt_device.cuh"
#include "owt_gpu.h"

namespace owt {

static_assert(kNoallocMaxNY == OWT_NOALLOC_MAX_NY, "table layout and the entry point's limit disagree");

constexpr int kNoallocThreads = 128;
constexpr size_t kNoallocSmem = 226 * 1024;

// Shared memory: tables, then the tile [row][line][component].
__host__ __device__ constexpr size_t noalloc_tables_bytes(int NY) { return (noalloc_setup_bytes(NY) + 15) / 16 * 16; }
constexpr size_t noalloc_smem(int NY, int lines) {
  return noalloc_tables_bytes(NY) + (size_t)NY * lines * sizeof(double2);
}
static_assert(noalloc_smem(kNoallocMaxNY, 1) <= kNoallocSmem, "the longest line does not fit");

__global__ void __launch_bounds__(kNoallocThreads)
    k_dy1_noalloc(int NY, int nlines, int tile, double alpha, const double2 *in, double2 *out) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int state[2];
  constexpr int KV = kNoallocKV;
  constexpr uint8_t kWide = 0x80;  // in piv: U has entries beyond two rows up in this column
  const NoallocSetup s = noalloc_layout(sm, NY);
  double2 *T = reinterpret_cast<double2 *>(sm + noalloc_tables_bytes(NY));
  const int t = threadIdx.x, line0 = blockIdx.x * tile;
  const int nl = nlines - line0 < tile ? nlines - line0 : tile;
  noalloc_assemble(s, NY, alpha, t, kNoallocThreads);
  __syncthreads();
  // B1 rows of the tile by all warps but the first, which factors A1 meanwhile
  for (int e = t - 32; e >= 0 && e < NY * nl; e += kNoallocThreads - 32) {
    const int j = e / nl, l = e - j * nl;
    double2 acc = make_double2(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double b = s.bval[j * 5 + q];
      const double2 f = in[(size_t)s.bcol[j * 5 + q] * nlines + line0 + l];
      if (nonzero(b)) {
        acc.x += b * f.x;
        acc.y += b * f.y;
      }
    }
    T[j * tile + l] = acc;
  }
  noalloc_factor_block(s, NY, t, kNoallocThreads, state, [] { __syncthreads(); });
  for (int j = t; j < NY; j += kNoallocThreads)
    if (nonzero(s.ab[j]) || nonzero(s.ab[NY + j])) s.piv[j] |= kWide;
  __syncthreads();
  // the band solve, one thread per line and component, in place
  if (t < 2 * nl) {
    double *x = reinterpret_cast<double *>(T) + t;
    const int ld = 2 * tile;
    {
      double w0 = x[0], w1 = x[ld], w2 = x[2 * ld];
#pragma unroll 4
      for (int j = 0; j < NY; ++j) {
        const int off = s.piv[j] & 3;
        if (off == 1) {
          const double q = w0; w0 = w1; w1 = q;
        } else if (off == 2) {
          const double q = w0; w0 = w2; w2 = q;
        }
        x[j * ld] = w0;
        const double y = w0;
        w0 = w1 - s.ab[(KV + 1) * NY + j] * y;
        w1 = w2 - s.ab[(KV + 2) * NY + j] * y;
        w2 = j + 3 < NY ? x[(j + 3) * ld] : 0.0;
      }
    }
    {
      auto at = [&](int j) { return j >= 0 ? x[j * ld] : 0.0; };
      double w0 = x[(NY - 1) * ld], w1 = at(NY - 2), w2 = at(NY - 3), w3 = at(NY - 4), w4 = at(NY - 5);
#pragma unroll 4
      for (int j = NY - 1; j >= 0; --j) {
        const double v = w0 * s.ab[KV * NY + j];
        x[j * ld] = v;
        w0 = w1 - s.ab[(KV - 1) * NY + j] * v;
        w1 = w2 - s.ab[(KV - 2) * NY + j] * v;
        w2 = w3;
        w3 = w4;
        if (s.piv[j] & kWide) {
          w2 -= s.ab[NY + j] * v;
          w3 -= s.ab[j] * v;
        }
        w4 = at(j - 5);
      }
    }
  }
  __syncthreads();
  for (int e = t; e < NY * nl; e += kNoallocThreads) {
    const int j = e / nl, l = e - j * nl;
    const double c = s.c11[j];
    const double2 d = T[j * tile + l];
    out[(size_t)j * nlines + line0 + l] = make_double2(c * d.x, c * d.y);
  }
}

}  // namespace owt

// capi.cu: the calling thread's message for owt_last_error(NULL)
void owt_set_thread_error(const std::string &m);

namespace {
// Per device: its SMs, and whether the kernel's shared-memory limit is raised
// there (once per device, with that device current).
std::mutex g_noalloc_mu;
int g_noalloc_sms[256] = {0};
}  // namespace

extern "C" int owt_dy1_noalloc(int64_t NY, int64_t nlines, double alpha_mesh, const double *d_in, double *d_out,
                               void *stream) {
  using namespace owt;
  auto fail = [&](int code, const std::string &m) {
    owt_set_thread_error(m);
    return code;
  };
  if (NY < 7 || NY > OWT_NOALLOC_MAX_NY)
    return fail(OWT_ERR_INVALID, "NY must be within [7, " + std::to_string(OWT_NOALLOC_MAX_NY) + "]");
  if (nlines < 1 || NY * nlines > (int64_t)OWT_NOALLOC_MAX_VALUES)
    return fail(OWT_ERR_INVALID, "NY * nlines must be within [1, " + std::to_string(OWT_NOALLOC_MAX_VALUES) +
                                     "] complex values");
  if (!(alpha_mesh > 0)) return fail(OWT_ERR_INVALID, "alpha_mesh must be positive");
  if (!d_in || !d_out || ((uintptr_t)d_in % 16) || ((uintptr_t)d_out % 16))
    return fail(OWT_ERR_INVALID, "d_in and d_out must be 16-byte aligned device pointers");
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 256) return fail(OWT_ERR_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
  int sms = 0;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_sms[dev]) {
      int n = 0;
      e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_dy1_noalloc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kNoallocSmem);
      if (e != cudaSuccess) return fail(OWT_ERR_CUDA, std::string("kernel attributes: ") + cudaGetErrorString(e));
      g_noalloc_sms[dev] = n > 0 ? n : 1;
    }
    sms = g_noalloc_sms[dev];
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int fits = (int)((kNoallocSmem - noalloc_tables_bytes((int)NY)) / ((size_t)NY * sizeof(double2)));
  const int tile = (int)std::min<int64_t>({(nlines + sms - 1) / sms, fits, kNoallocThreads / 2});
  k_dy1_noalloc<<<(unsigned)((nlines + tile - 1) / tile), kNoallocThreads, noalloc_smem((int)NY, tile), st>>>(
      (int)NY, (int)nlines, tile, alpha_mesh, reinterpret_cast<const double2 *>(d_in),
      reinterpret_cast<double2 *>(d_out));
  e = cudaGetLastError();
  if (e != cudaSuccess) return fail(OWT_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(e));
  return OWT_OK;
}
