// Products, sums and differences of the FP64 kernels, plain or as three-register
// multiply-adds.
#pragma once

#include <cuda_runtime.h>

namespace hg {

// With four or more warps on an SM its FP64 unit takes a multiply, an add, or a
// fused multiply-add with a constant operand every 19.0 cycles, but a fused
// multiply-add of three registers every 16.0 (measured, 4 to 32 warps); one warp
// alone waits 63.1 and 64.6.  So the kernels and layouts that fill the unit form
// them as fused multiply-adds with a neutral operand: a b + (-0), a 1 + b and
// (-b) 1 + a round once and have the bits of a * b, a + b and a - b, signed zeros
// included.  The neutral operands come by volatile loads: the compiler would
// fold known ones back.
struct PlainOps {
  __device__ __forceinline__ double mul(double a, double b) const { return a * b; }
  __device__ __forceinline__ double add(double a, double b) const { return a + b; }
  __device__ __forceinline__ double sub(double a, double b) const { return a - b; }
};
__device__ static double hg_neutral[2] = {1.0, -0.0};
struct FusedOps {
  double one, nz;
  __device__ __forceinline__ FusedOps() {
    asm volatile("ld.volatile.global.f64 %0, [%1];" : "=d"(one) : "l"(hg_neutral));
    asm volatile("ld.volatile.global.f64 %0, [%1];" : "=d"(nz) : "l"(hg_neutral + 1));
  }
  __device__ __forceinline__ double mul(double a, double b) const { return fma(a, b, nz); }
  __device__ __forceinline__ double add(double a, double b) const { return fma(a, one, b); }
  __device__ __forceinline__ double sub(double a, double b) const { return fma(-b, one, a); }
};

}  // namespace hg
