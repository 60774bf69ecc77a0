// Checks the device forms of hg_exact.cuh (hg_sqrt, hg_div, hg_quotients with
// the hardware's FP32 estimates) against IEEE sqrt and division and, for
// hg_quotients, the hg_div_rn sequence: random significands, binade edges,
// exponents in and out of the accepted range, zero numerators.  Prints
// "<samples> <wrong> <error>".  Bounded grid-stride loop, one atomic counter.
#include <cstdio>
#include <cstdlib>
#include <cuda_runtime.h>
#include "hg_exact.cuh"

__device__ unsigned long long mix(unsigned long long x) {
  x ^= x >> 33; x *= 0xff51afd7ed558ccdull; x ^= x >> 33; x *= 0xc4ceb9fe1a85ec53ull; x ^= x >> 33;
  return x;
}
__device__ double make(unsigned long long r, int mode, bool negative) {
  unsigned long long mant = r & 0x000FFFFFFFFFFFFFull;
  if (mode == 1) mant = 0x000FFFFFFFFFFFFFull - (r & 0xFF);
  if (mode == 2) mant = r & 0xFF;
  const int span = (r >> 60) == 0 ? 480 : 60;
  const unsigned long long e = 1023 - span + (unsigned long long)((r >> 40) % (2 * span));
  return __longlong_as_double((long long)((negative ? 1ull << 63 : 0ull) | (e << 52) | mant));
}
__device__ bool differ(double a, double b) { return __double_as_longlong(a) != __double_as_longlong(b); }
__global__ void check(unsigned long long n, unsigned long long seed, unsigned long long* bad) {
  unsigned long long local = 0;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long r0 = mix(i * 4 + seed), r1 = mix(i * 4 + 1 + seed), r2 = mix(i * 4 + 2 + seed * 7),
                             r3 = mix(i * 4 + 3 + seed * 3);
    const double d = make(r0, (int)(i % 3), false);
    double num[3] = {make(r1, (int)((i / 3) % 3), r2 & 1), make(r2, 0, r1 & 1), make(r3, 0, r0 & 1)};
    if (i % 11 == 0) num[i % 3] = (r3 & 2) ? -0.0 : 0.0;
    double q[3];
    hg_quotients(num, d, q);
    const double rd = hg_rcp_rn(d);
    for (int k = 0; k < 3; ++k) local += differ(q[k], hg_div_rn(num[k], d, rd));
    local += differ(hg_sqrt(d), __dsqrt_rn(d));
    const double v = hg_div(num[0], d), w = __ddiv_rn(num[0], d);
    local += differ(v, w);
  }
  if (local) atomicAdd(bad, local);
}
int main(int argc, char** argv) {
  const unsigned long long n = argc > 1 ? strtoull(argv[1], 0, 10) : (1ull << 28);
  unsigned long long *bad, h = 1;
  if (cudaMalloc(&bad, 8) != cudaSuccess || cudaMemset(bad, 0, 8) != cudaSuccess) return 1;
  check<<<152 * 8, 256>>>(n, 12345, bad);
  cudaMemcpy(&h, bad, 8, cudaMemcpyDeviceToHost);
  const cudaError_t e = cudaGetLastError();
  printf("%llu %llu %s\n", n, h, cudaGetErrorName(e));
  cudaFree(bad);
  return e == cudaSuccess ? 0 : 1;
}
