// DevBuf over an allocator that refuses: no buffer may look larger than it is.
#include "dev_buf.h"

#include <cstdio>
#include <cstdlib>

static int g_refuse = 0, g_live = 0;
static cudaError_t g_last = cudaSuccess;

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  if (g_refuse > 0) {
    --g_refuse;
    *p = reinterpret_cast<void*>(0x10);  // what a failed call leaves there is not to be used
    return g_last = cudaErrorMemoryAllocation;
  }
  *p = std::malloc(n);
  ++g_live;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::free(p);
  --g_live;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
}

static int failures = 0;
#define CHECK(x) \
  if (!(x)) std::printf("line %d: %s\n", __LINE__, #x), ++failures

int main() {
  {
    lai::host::DevBuf b;
    g_refuse = 1;
    CHECK(b.ensure(64) == cudaErrorMemoryAllocation);
    CHECK(b.p == nullptr && b.bytes == 0);
    CHECK(cudaGetLastError() == cudaSuccess);
    CHECK(b.ensure(64) == cudaSuccess && b.p && b.bytes == 64);
    CHECK(b.ensure(32) == cudaSuccess && b.bytes == 64);
    g_refuse = 1;  // growing frees the old buffer first
    CHECK(b.ensure(128) == cudaErrorMemoryAllocation);
    CHECK(b.p == nullptr && b.bytes == 0);
    CHECK(b.ensure(16) == cudaSuccess && b.p && b.bytes == 16);
    CHECK(b.alloc(0) == cudaSuccess && b.p == nullptr && b.bytes == 0);
  }
  CHECK(g_live == 0);
  std::printf("%d failures\n", failures);
  return failures != 0;
}
