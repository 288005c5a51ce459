// Host arrays that kernels read and write directly: the whole array has to lie
// in one allocation or registration of page-locked memory that the GPU may
// access so.  (An array registered in part, or in several pieces, has bytes the
// GPU must not touch although its first and last ones are page-locked.)
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace owt {

// What the driver says about an array's first byte.
struct HostRange {
  bool pinned = false;             // page-locked host memory with a device address
  uintptr_t start = 0;             // of the allocation or registration
  size_t size = 0;
  bool readable = false, writable = false;  // by kernels
  uintptr_t device = 0;            // device address of the first byte
};

// Device address of bytes [p, p + bytes), or null where kernels may not access
// all of them; 16-byte aligned (the kernels move 16 bytes at a time).
inline void *host_view(const HostRange &r, uintptr_t p, size_t bytes, bool write) {
  if (!r.pinned || p % 16 != 0 || r.device % 16 != 0) return nullptr;
  if (p < r.start || p - r.start > r.size || bytes > r.size - (p - r.start)) return nullptr;
  if (!r.readable || (write && !r.writable)) return nullptr;
  return reinterpret_cast<void *>(r.device);
}

inline HostRange host_range(const void *p) {
  using Query = CUresult (*)(unsigned, CUpointer_attribute *, void **, CUdeviceptr);
  static const Query query = [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &f, 12000, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      return static_cast<Query>(nullptr);
    }
    return reinterpret_cast<Query>(f);
  }();
  HostRange r;
  cudaPointerAttributes at{};
  auto attributes = [&] {
    if (cudaPointerGetAttributes(&at, p) == cudaSuccess) return at.type == cudaMemoryTypeHost;
    cudaGetLastError();
    return false;
  };
  if (!query || !attributes()) return r;
  int dev = 0;
  // no device address where the device is not current in this thread yet
  if (!at.devicePointer && !(cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess && attributes()))
    return r;
  if (!at.devicePointer) return r;
  CUdeviceptr start = 0;
  size_t size = 0;
  unsigned long long access = 0;
  CUpointer_attribute what[] = {CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE,
                                CU_POINTER_ATTRIBUTE_ACCESS_FLAGS};
  void *data[] = {&start, &size, &access};
  if (query(3, what, data, reinterpret_cast<CUdeviceptr>(p)) != CUDA_SUCCESS) return r;
  r.pinned = true;
  // (a range is given by its device addresses; host and device addresses
  // differ by the same offset throughout it)
  r.device = reinterpret_cast<uintptr_t>(at.devicePointer);
  r.start = (uintptr_t)start + (reinterpret_cast<uintptr_t>(p) - r.device);
  r.size = size;
  r.readable = access == CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READ || access == CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READWRITE;
  r.writable = access == CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READWRITE;
  return r;
}

}  // namespace owt
