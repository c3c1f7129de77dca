// FP64 reciprocals on the chains of dependent steps, where CUDA's division (its own reciprocal, a
// correction and a branch on the range) takes two to three times as long: with two divisions, or a
// branch to one, an iteration of the resident PCG took 1 to 2% longer (64 x 64 grid, one solve: 1.190
// -> 1.214 and 1.197 ms).
#pragma once

namespace mg {

// 1 / v by two Newton steps on the hardware's approximation, each of which doubles the correct bits:
// within a unit in the last place of 1.0 / v for |v| in [2^-1000, 2^1000]. NaN for zeros,
// subnormals and infinities.
__device__ __forceinline__ double recip(double v) {
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(v));
  x = fma(x, fma(-v, x, 1.0), x);
  return fma(x, fma(-v, x, 1.0), x);
}

// a / v where |v| is infinite or in recip()'s range; NaN for a NaN
__device__ __forceinline__ double quotient(double a, double v) {
  return a * ((__double2hiint(v) & 0x7fffffff) == 0x7ff00000 ? 0.0 : recip(v));
}

}  // namespace mg
