// Device memory owned by an object of the host side.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace lai {
namespace host {

struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() { if (p) cudaFree(p); }
  // A new buffer of n bytes in the place of the old one; none after a failure.
  cudaError_t alloc(size_t n) {
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
    if (n == 0) return cudaSuccess;
    const cudaError_t e = cudaMalloc(&p, n);
    if (e != cudaSuccess) {
      p = nullptr;
      cudaGetLastError();  // reported here: a later launch check must not find it
      return e;
    }
    bytes = n;
    return cudaSuccess;
  }
  // At least n bytes (contents are lost where it grows).
  cudaError_t ensure(size_t n) { return bytes >= n ? cudaSuccess : alloc(n); }
  template <typename T> T* as() const { return static_cast<T*>(p); }
};

}  // namespace host
}  // namespace lai
