// 1/sqrt(x) in FP64 for the pair kernels: the hardware's estimate
// (rsqrt.approx.ftz.f64) and one step of Halley's third-order iteration,
//   e = 1 - x y^2,   y <- y + y e (1/2 + 3/8 e),
// whose error is 5/16 e^3: from an estimate good to 2^-20 full FP64 precision
// in five FMA-pipe operations.  The estimate's lower 32 bits are zero, so y^2
// is exact and e carries one rounding, of its own small size: 0.507 units in the
// last place at most over 16 million arguments, as CUDA's rsqrt.  For 0, infinite
// or NaN x the result is NaN (a pair at distance 0 has no finite rates either
// way), for positive subnormal x infinity; rsqrt_f64_full gives 0 for infinity (a
// distance whose square overflows) and infinity for 0 too, two integer operations
// and a select more.
#pragma once

namespace pawan {

__device__ __forceinline__ double rsqrt_f64(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y * y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

__device__ __forceinline__ double rsqrt_f64_full(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y * y, 1.0);
  const double r = fma(y * e, fma(0.375, e, 0.5), y);
  // a positive normal estimate is refined, 0 and infinity are the result
  return (unsigned)(__double2hiint(y) - 0x00100000) < 0x7fe00000u ? r : y;
}

}  // namespace pawan
