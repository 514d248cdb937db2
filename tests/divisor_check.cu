// k_check_prepared (arith_check.cu) on a table of divisors that the caller
// prepared.
#include "arith_check.cu"

extern "C" int divisor_check(unsigned long long n, unsigned long long seed, const hc_divisor* h,
                             int ntab, unsigned long long* bad, double* first) {
  hc_divisor* tab;
  unsigned long long* d_bad;
  double* d_first;
  if (cudaMalloc(&tab, ntab * sizeof(hc_divisor)) != cudaSuccess ||
      cudaMalloc(&d_bad, 8) != cudaSuccess || cudaMalloc(&d_first, 32) != cudaSuccess)
    return 1;
  cudaMemcpy(tab, h, ntab * sizeof(hc_divisor), cudaMemcpyHostToDevice);
  cudaMemset(d_bad, 0, 8);
  cudaMemset(d_first, 0, 32);
  k_check_prepared<<<152 * 16, 256>>>(n, seed, tab, ntab, d_bad, d_first);
  cudaMemcpy(bad, d_bad, 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(first, d_first, 32, cudaMemcpyDeviceToHost);
  const cudaError_t e = cudaGetLastError();
  cudaFree(tab);
  cudaFree(d_bad);
  cudaFree(d_first);
  return e == cudaSuccess ? 0 : 2;
}
