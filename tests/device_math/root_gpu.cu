// Compares root_rn (csrc/projector.cuh) with the IEEE square root on the GPU
// for every float of its range -- TEST INFRASTRUCTURE.
#include "../../asd_pocs_mex_cuda_demo_gb300/csrc/projector.cuh"

__global__ void k_root(unsigned lo, unsigned hi, unsigned long long *bad) {
  unsigned long long n = 0;
  for (unsigned long long b = lo + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
       b <= hi; b += (unsigned long long)gridDim.x * blockDim.x) {
    const float x = __uint_as_float((unsigned)b);
    n += __float_as_uint(asd::root_rn(x)) != __float_as_uint(sqrtf(x));
  }
  if (n) atomicAdd(bad, n);
}

// Floats with bit patterns lo .. hi whose roots differ; negative on an error.
extern "C" long long root_mismatches(unsigned lo, unsigned hi) {
  unsigned long long *d = nullptr, n = 0;
  if (cudaMalloc(&d, sizeof n) != cudaSuccess) return -1;
  cudaMemset(d, 0, sizeof n);
  k_root<<<152 * 8, 256>>>(lo, hi, d);
  const cudaError_t e = cudaMemcpy(&n, d, sizeof n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? (long long)n : -2;
}
extern "C" float root_min() { return asd::kRootMin; }
