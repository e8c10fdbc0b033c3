// DevBuf against a CUDA runtime that is out of memory for the first argv[2] allocations. argv[1]:
// pooled or plain; argv[3]: retried (the allocation succeeds after the pools were trimmed) or refused
// (ORION_ERR_NOMEM, and no error left for the next call to find).
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "context.h"

namespace {
int g_failures = 0, g_trims = 0, g_mallocs = 0;
cudaError_t g_last = cudaSuccess;
char g_memory[64];

cudaError_t allocate(void** p) {
  ++g_mallocs;
  if (g_failures > 0) {
    --g_failures;
    *p = nullptr;
    return g_last = cudaErrorMemoryAllocation;
  }
  *p = g_memory;
  return cudaSuccess;
}
}  // namespace

extern "C" {
cudaError_t cudaMalloc(void** p, size_t) { return allocate(p); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t, cudaMemPool_t, cudaStream_t) { return allocate(p); }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaFreeAsync(void*, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "out of memory"; }
}

namespace orion_gb300 {
int fail(int code, const std::string&) { return code; }
void trim_scene_pools() { ++g_trims; }
}  // namespace orion_gb300

int main(int, char** argv) {
  orion_gb300::DevBuf b;
  g_failures = std::atoi(argv[2]);
  const int rc = std::strcmp(argv[1], "pooled") == 0 ? b.alloc_pooled(48, nullptr, reinterpret_cast<cudaStream_t>(1))
                                                     : b.alloc(48);
  if (std::strcmp(argv[3], "retried") == 0) {
    if (rc != ORION_OK || g_trims != 1 || g_mallocs != 2 || b.p != g_memory || b.bytes != 48)
      return std::printf("rc %d after %d trims\n", rc, g_trims), 1;
  } else {
    if (rc != ORION_ERR_NOMEM || b.p || b.bytes) return std::printf("rc %d\n", rc), 1;
  }
  if (cudaGetLastError() != cudaSuccess) return std::puts("an error is left behind"), 1;
  std::puts("ok");
  return 0;
}
