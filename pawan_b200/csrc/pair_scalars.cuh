// FP32 pair scalars shared by the one-sided (pair_f32.cu) and the symmetric
// (pair_sym.cu) pair kernels: q, F and the diffusion factor of a pair in the
// formulations of the tile-pair classes, the accurate cross product, and the
// tiles' box geometry.
#pragma once

#include "device.cuh"

namespace pawan {
namespace {

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// q, F and the diffusion factor of one pair in units of A = 1/(4 pi), from
// sigma^2, w = (rho^2 + sigma^2)^-1/2 and ri = 1/rho (u = sigma^2 w^2):
//   Dp = (u w)^5 = sigma^10 w^15,  Zc = Dp sigma^2,
//   ph = (rho^2 + 1.5 sigma^2) w^4 / rho = (1 + u/2) w^2 / rho,
//   qh = (ph - 7.5 Zc) sigma^2 / rho^2,   fh = (2.5 Zc - qh) / rho^2.
// 16 FP32 instructions.
__device__ __forceinline__ void kernel_scalars(float sig2, float w, float ri, float &qh, float &fh,
                                               float &dp) {
  const float w2 = w * w;
  const float uu = sig2 * w2;
  const float v = uu * w;
  const float v2 = v * v;
  const float v4 = v2 * v2;
  dp = v4 * v;
  const float zc = dp * sig2;
  const float ph = fmaf(0.5f, uu, 1.0f) * w2 * ri;
  const float ri2 = ri * ri;
  qh = fmaf(-7.5f, zc, ph) * sig2 * ri2;
  fh = fmaf(2.5f, zc, -qh) * ri2;
}

// kernel_scalars for sigma^2 = 2h the same for every pair of the tile, with
// the factors that do not vary per pair left to the per-tile fold: returns
//   qs = qh / sigma^2,  fs = fh / sigma^2,  ds = Dp / 32,
// from u' = h w^2 = u/2 and v' = u' w = v/2 (so ds = v'^5):
//   ph = (1 + u') w^2 / rho,  qs = (ph - 240 sigma^2 ds) / rho^2,
//   fs = (80 ds - qs) / rho^2.
// 1/rho^2 comes from the MUFU reciprocal; 12 FP32 instructions.
__device__ __forceinline__ void kernel_scalars_uniform(float h, float c240, float w, float ri,
                                                       float r2, float &qs, float &fs, float &ds) {
  const float y = w * w;
  const float u = h * y;
  const float v = u * w;
  const float v2 = v * v;
  ds = v2 * v2 * v;
  const float ph = fmaf(u, y, y) * ri;
  const float ri2 = rcp_approx(r2);
  qs = fmaf(c240, ds, ph) * ri2;
  fs = fmaf(80.f, ds, -qs) * ri2;
}

// The same with 1/rho^2 from rsqrt squared instead of a MUFU reciprocal.
__device__ __forceinline__ void kernel_scalars_uniform(float h, float c240, float w, float ri, float &qs,
                                                       float &fs, float &ds) {
  const float y = w * w;
  const float u = h * y;
  const float v = u * w;
  const float v2 = v * v;
  ds = v2 * v2 * v;
  const float ph = fmaf(u, y, y) * ri;
  const float ri2 = ri * ri;
  qs = fmaf(c240, ds, ph) * ri2;
  fs = fmaf(80.f, ds, -qs) * ri2;
}

// Far field without the Z terms.  Where every pair of a tile pair has
// rho >= 6 sigma (checked on the tiles' boxes), Z = (15/8pi) sigma^-3
// (rho_bar^2 + 1)^-7.5 is below 3e-9 of phi/rho_bar in q = (phi/rho_bar - Z)
// / rho_bar^2 and of 3q in F = (Z - 3q)/rho^2, i.e. twenty times below FP32
// rounding, and the diffusion rate 2 nu Z / sigma^2 (v_i alpha_j - v_j alpha_i)
// of those pairs is as small against the near-field diffusion: the terms are
// zero at FP32 resolution and are not formed.  What remains, with
// y = 1/(rho^2 + sigma^2) and (rho^2 + 1.5 sigma^2) w^4 = y (1 + y sigma^2/2):
//   qh = y (1 + y sigma^2/2) sigma^2 / rho^3,   fh = -qh / rho^2.
// kernel_scalars_nz returns them for one sigma^2 per pair (12 FP32
// instructions with the MUFU reciprocal and rsqrt); the uniform-radius form
// returns qs = qh / sigma^2, -fs = qh / (sigma^2 rho^2) (8 instructions).
__device__ __forceinline__ void kernel_scalars_nz(float sig2, float r2, float &qh, float &nfh) {
  const float y = rcp_approx(r2 + sig2);
  const float ri = rsqrtf(r2);
  const float ri2 = ri * ri;
  const float hy = 0.5f * sig2 * y;
  const float ph = fmaf(hy, y, y);
  qh = ph * sig2 * ri * ri2;
  nfh = qh * ri2;
}

// Far field without the Z terms, and a series for the smoothing factor.
// With eps = sigma^2 / rho^2,
//   rho^2 y (1 + y sigma^2/2) = 1/(1 + eps) + (eps/2)/(1 + eps)^2
//                             = 1 - eps/2 + 0 eps^2 + eps^3/2 - ...,
// so where every pair of a tile pair has rho >= 16 sigma (eps <= 1/256, checked
// on the tiles' boxes) the two-term form 1 - sigma^2/(2 rho^2) is exact to
// 3.0e-8 relative, below FP32's unit roundoff (6e-8):
//   qh = sigma^2 rho^-5 (1 - sigma^2 rho^-2 / 2),   fh = -qh / rho^2,
// one MUFU rsqrt per pair instead of an rsqrt and a reciprocal (the
// uniform-radius form returns qs = qh / sigma^2 = rho^-5 (1 - h rho^-2)).
__device__ __forceinline__ void kernel_scalars_series(float sig2, float r2, float &qh, float &nfh) {
  const float ri = rsqrtf(r2);
  const float ri2 = ri * ri;
  const float e = sig2 * ri2;
  const float c = fmaf(-0.5f, e, 1.0f);
  qh = e * ri * ri2 * c;
  nfh = qh * ri2;
}

// The Gaussian kernel (gaussian.h:20-59) in the units of kernel_scalars: with
// x2 = rho^2/sigma^2, e = exp(-x2/2) and K = sqrt(2/pi),
//   qh = gq / sigma^3,        gq = (erf(x/sqrt 2)/x - K e) / x2,
//   fh = gf / (3 sigma^5),    gf = (K e - 3 gq) / x2,
//   dp = (2/15) K e / sigma^5.
// Below x2 = 1 the closed forms lose digits to cancellation; there gq and gf
// come from their power series in y = -x2/2,
//   gq = K sum_m y^m / (m! (2m+3)),   gf = -K sum_m y^m / (m! (2m+5)),
// nine terms (relative truncation error < 1e-8 at x2 = 1).
// Far field of the Gaussian kernel: where every pair of a tile pair
// has x = rho/sigma >= 7 (checked on the tiles' boxes), e = exp(-x2/2) <=
// 2.3e-11 and erf(x/sqrt 2) = 1 - 2.6e-12, so gq = 1/x^3 to 1.3e-10 relative
// (K e x against 1), gf = -3/x^5 to 2.1e-9 (K e x^3/3 against 1) and dp is 0
// at FP32 resolution:
//   qh = rho^-3,   fh = -rho^-5 = -qh / rho^2,   dp = 0,
// the singular field, one MUFU rsqrt and three multiplies per pair in place of
// an exp and an erf (the far loops' series branches with KERN = Gaussian).
__device__ __forceinline__ void gauss_scalars(float sig2, float r2, float ri, float &qh, float &fh,
                                              float &dp) {
  const float K = 0.797884561f;
  const float is = rsqrtf(sig2);
  const float is2 = is * is;
  const float is3 = is2 * is;
  const float x2 = r2 * is2;
  const float e = expf(-0.5f * x2);
  float gq, gf;
  if (x2 < 1.0f) {
    const float y = -0.5f * x2;
    float sq = 1.0f / (40320.0f * 19.0f), sf = 1.0f / (40320.0f * 21.0f);
    sq = fmaf(sq, y, 1.0f / (5040.0f * 17.0f));
    sf = fmaf(sf, y, 1.0f / (5040.0f * 19.0f));
    sq = fmaf(sq, y, 1.0f / (720.0f * 15.0f));
    sf = fmaf(sf, y, 1.0f / (720.0f * 17.0f));
    sq = fmaf(sq, y, 1.0f / (120.0f * 13.0f));
    sf = fmaf(sf, y, 1.0f / (120.0f * 15.0f));
    sq = fmaf(sq, y, 1.0f / (24.0f * 11.0f));
    sf = fmaf(sf, y, 1.0f / (24.0f * 13.0f));
    sq = fmaf(sq, y, 1.0f / (6.0f * 9.0f));
    sf = fmaf(sf, y, 1.0f / (6.0f * 11.0f));
    sq = fmaf(sq, y, 1.0f / (2.0f * 7.0f));
    sf = fmaf(sf, y, 1.0f / (2.0f * 9.0f));
    sq = fmaf(sq, y, 1.0f / 5.0f);
    sf = fmaf(sf, y, 1.0f / 7.0f);
    sq = fmaf(sq, y, 1.0f / 3.0f);
    sf = fmaf(sf, y, 1.0f / 5.0f);
    gq = K * sq;
    gf = -K * sf;
  } else {
    const float x = r2 * ri * is;  // rho / sigma
    const float ix = rcp_approx(x);
    const float ix2 = ix * ix;
    gq = fmaf(erff(0.707106781f * x), ix, -K * e) * ix2;
    gf = fmaf(-3.0f, gq, K * e) * ix2;
  }
  const float is5 = is3 * is2;
  qh = gq * is3;
  fh = gf * is5 * (1.0f / 3.0f);
  dp = (2.0f / 15.0f) * K * e * is5;
}

// (a + a_lo) x (b + b_lo) for a target strength a + a_lo and a source strength
// b + b_lo (FP32 hi + lo), accurate to a few ulp of the result also for nearly
// parallel or antiparallel strengths, in 19 operations (cross_accurate: 27).
// With mu = (a.b)/|a|^2, v = b - mu a is formed by one FMA per component, so
// exactly up to its own rounding, and a x v = a x b whatever mu's rounding
// (its error only moves v along a).  v is (nearly) perpendicular to a, so
// a x (v + b_lo) has no cancellation; and a_lo x b = mu (a_lo x a) + a_lo x v,
// the last term eps |a||v| relative to |a x v| = |a||v|.  iaa = 1/|a|^2 (0
// for a = 0) and (lx, ly, lz) = a_lo x a are per target.
// Also returns mu and v + b_lo: b + b_lo = mu a + (v + b_lo).
__device__ __forceinline__ void projection_cross(float ax, float ay, float az, float iaa, float lx,
                                                 float ly, float lz, float bx, float by, float bz,
                                                 float mx, float my, float mz, float &wx, float &wy,
                                                 float &wz, float &mu, float &vx, float &vy, float &vz) {
  mu = fmaf(az, bz, fmaf(ay, by, ax * bx)) * iaa;
  vx = fmaf(-mu, ax, bx) + mx;
  vy = fmaf(-mu, ay, by) + my;
  vz = fmaf(-mu, az, bz) + mz;
  wx = fmaf(mu, lx, fmaf(ay, vz, -az * vy));
  wy = fmaf(mu, ly, fmaf(az, vx, -ax * vz));
  wz = fmaf(mu, lz, fmaf(ax, vy, -ay * vx));
}

__device__ __forceinline__ float box_gap2(float4 alo, float4 ahi, float4 blo, float4 bhi) {
  const float gx = fmaxf(0.f, fmaxf(alo.x - bhi.x, blo.x - ahi.x));
  const float gy = fmaxf(0.f, fmaxf(alo.y - bhi.y, blo.y - ahi.y));
  const float gz = fmaxf(0.f, fmaxf(alo.z - bhi.z, blo.z - ahi.z));
  return gx * gx + gy * gy + gz * gz;
}

// Squared half-diagonal of a box.
__device__ __forceinline__ float box_half_diag2(float4 lo, float4 hi) {
  const float ex = hi.x - lo.x, ey = hi.y - lo.y, ez = hi.z - lo.z;
  return 0.25f * (ex * ex + ey * ey + ez * ez);
}

}  // namespace
}  // namespace pawan
