// host_cudart.cpp -- a stand-in for the CUDA runtime in host tests of launch
// and planning code: device memory is host memory, launches do nothing.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
  *p = std::malloc(n);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void *p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st *) { return 1; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t *, const void *) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void **, size_t, cudaStream_t) { return cudaSuccess; }
void **__cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {}
}
