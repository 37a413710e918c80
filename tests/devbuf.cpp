// CPU check of DevBuf (csrc/common.hpp) against a CUDA runtime that is out of
// memory: the runtime's functions are fakes in this file.
#include <cstdio>
#include <cstdlib>

#include "common.hpp"

static bool out_of_memory = false;

extern "C" {
cudaError_t cudaMalloc(void **p, size_t bytes) {
  if (out_of_memory) return cudaErrorMemoryAllocation;
  *p = std::malloc(bytes);
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaMemcpyAsync(void *, const void *, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
}

int main() {
  rchol::DevBuf<double> fresh, grown(4);
  out_of_memory = true;
  for (rchol::DevBuf<double> *b : {&fresh, &grown}) {
    int status = 0;
    try {
      b->alloc(8);
    } catch (const rchol::Error &e) {
      status = e.status;
    }
    if (status != RCHOL_ERR_NOMEM || b->p || b->n != 0) {
      std::printf("FAIL status %d p %p n %zu\n", status, (void *)b->p, b->n);
      return 1;
    }
  }
  out_of_memory = false;
  fresh.alloc(8);
  if (!fresh.p || fresh.n != 8) return 1;
  std::printf("ok\n");
  return 0;
}
