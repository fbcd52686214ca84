// All-pairs interaction in FP64 with the kernel algebra of the FP32 kernel
// (pair_f32.cu): two rsqrt per pair, no pow, no division; alpha_i x alpha_j
// per pair as the reference forms it.  (Forming the stretching's q-term as
// alpha_i x sum(q alpha_j) and the triple product from the velocity's cross
// product as well saves six more operations per pair but sums nearly parallel
// neighbours' terms coherently before the cross product: 100 times the rounding
// error of the per-pair form.)  This is the "tuned FP64" variant, reported
// beside the FP32 kernel and the plain FP64 comparator (pair_plain.cu).
//
// Reference: INTERACT (src/interaction/interaction_utils.h:363-407), KERNEL
// (src/interaction/highorder.h:48-60), __interaction::interact
// (src/interaction/interaction.cpp:95-108).  The Gaussian kernel
// (src/interaction/gaussian.h:20-59) in the same units: with x2 = rho^2/sigma^2,
// e = exp(-x2/2), K = sqrt(2/pi), gq = (erf(x/sqrt 2)/x - K e)/x2 and
// gf = (K e - 3 gq)/x2: qh = gq/sigma^3, fh = gf/(3 sigma^5),
// dp = (2/15) K e / sigma^5 (closed forms, as the reference evaluates them).
//
// Runs on the symmetric pair engine (pair_sym.cuh), each unordered pair once:
// q (alpha_j x d) for the target and -q (alpha_i x d) for the source, and one
// vector s = q (alpha_i x alpha_j) + 3 F t d + 15 nu Dp (v_i alpha_j - v_j alpha_i)
// that is added to one and taken from the other.  As in the FP32 kernel a
// lane's targets stay in registers and 32 sources in shared memory, whose six
// sums travel by shuffle.  Bound by the FP64 pipe: 87 operations for two
// interactions (77 without diffusion) against 76 for one before.  One
// right-hand side on one B200: ring pair at N = 65,536 12.2 ms (352 G
// interactions/s, 0.83 of the pipe) against 19.3; at N = 2,048 27 us against 69.
#include "pair_sym.cuh"
#include "rsqrt64.cuh"

namespace pawan {
namespace {

constexpr int kStage64 = 4 * 512;    // per warp: 4 x double2[32]
// Targets per lane and blocks per SM: four targets in 255 registers keep the
// FP64 pipe fullest (one right-hand side of the ring pair at N = 16,384: 0.787
// ms, against 0.819 with two targets and three blocks, 0.865 with one and four);
// the Gaussian kernel's exp and erf want the warps instead (1.89 ms at N =
// 16,000 with one and four, 2.05 with two and three, 2.52 with four and two).
template <int KERN>
struct Shape64 {
  static constexpr int targets = KERN == KERNEL_GAUSSIAN ? 1 : 4;
  static constexpr int blocks = KERN == KERNEL_GAUSSIAN ? 4 : 2;
};

// Particles past the end: far away on opposite sides, with zero strength and
// volume, so that every term they enter is exactly zero.
constexpr double kPad64 = 1e150;

// Gaussian qh, fh, dp (see the file comment) from r2, sig2 and 1/rho.
__device__ __forceinline__ void gauss_f64(double r2, double sig2, double ri, double &qh,
                                          double &fh, double &dp) {
  const double is = rsqrt_f64(sig2);
  const double is2 = is * is;
  const double is3 = is2 * is;
  const double x2 = r2 * is2;
  const double e = exp(-0.5 * x2);
  const double x = r2 * ri * is;
  const double gq = (erf(kSqrtHalf * x) / x - kSqrt2OverPi * e) / x2;
  const double gf = (kSqrt2OverPi * e - 3.0 * gq) / x2;
  qh = gq * is3;
  fh = gf * is3 * is2 / 3.0;
  dp = (2.0 / 15.0) * kSqrt2OverPi * e * is3 * is2;
}

struct Sums64 {
  double ux, uy, uz, sx, sy, sz;
};

__device__ __forceinline__ void rotate(Sums64 &a, int m) {
  a.ux = __shfl_xor_sync(kFull, a.ux, m);
  a.uy = __shfl_xor_sync(kFull, a.uy, m);
  a.uz = __shfl_xor_sync(kFull, a.uz, m);
  a.sx = __shfl_xor_sync(kFull, a.sx, m);
  a.sy = __shfl_xor_sync(kFull, a.sy, m);
  a.sz = __shfl_xor_sync(kFull, a.sz, m);
}

__device__ __forceinline__ void add64(const Sums64 &s, double f, double *acc) {
  acc[0] += f * s.ux;
  acc[kT] += f * s.uy;
  acc[2 * kT] += f * s.uz;
  acc[3 * kT] += f * s.sx;
  acc[4 * kT] += f * s.sy;
  acc[5 * kT] += f * s.sz;
}

// DIAG: tile I against itself; every ordered pair is visited and only the
// targets' sums are kept.
template <int SIDE, bool DIAG, bool DIFF, int KERN>
__device__ __forceinline__ void pairs64(const SymSeg &sg, int I, int J, int k0, int k1, char *stage, int lane,
                                        double *accI, double *accJ) {
  constexpr int kR = Shape64<KERN>::targets;
  double2 *const s0 = reinterpret_cast<double2 *>(stage);  // x, y
  double2 *const s1 = s0 + 32;                             // z, s^2 / 2
  double2 *const s2 = s1 + 32;                             // alpha x, y
  double2 *const s3 = s2 + 32;                             // alpha z, volume
  const int n = sg.n;
  const double kap = 15.0 * sg.nu;
#pragma unroll 1
  for (int t0 = 0; t0 < kT; t0 += 32 * kR) {
    double4 p[kR], a[kR];  // w: s^2 / 2, volume
    Sums64 sum[kR];
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const int i = I * kT + t0 + 32 * r + lane;
      p[r] = make_double4(-kPad64, -kPad64, -kPad64, 1.0);
      a[r] = make_double4(0.0, 0.0, 0.0, 0.0);
      if (i < n) {
        p[r] = sg.pos64[i];
        a[r] = sg.vor64[i];
        p[r].w = 0.5 * p[r].w * p[r].w;
      }
      sum[r] = Sums64{0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    }
#pragma unroll 1
    for (int k = k0; k < k1; ++k) {
      const int j = J * kT + 32 * k + lane;
      double4 pj = make_double4(kPad64, kPad64, kPad64, 1.0), aj = make_double4(0.0, 0.0, 0.0, 0.0);
      if (j < n) {
        pj = sg.pos64[j];
        aj = sg.vor64[j];
        pj.w = 0.5 * pj.w * pj.w;
      }
      s0[lane] = make_double2(pj.x, pj.y);
      s1[lane] = make_double2(pj.z, pj.w);
      s2[lane] = make_double2(aj.x, aj.y);
      s3[lane] = make_double2(aj.z, aj.w);
      __syncwarp();
      const int self = k - t0 / 32;  // the target whose own pair falls on step 0
      Sums64 b{0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
      for (int m = 0; m < 32; ++m) {
        const double2 q0 = s0[lane ^ m], q1 = s1[lane ^ m], q2 = s2[lane ^ m], q3 = s3[lane ^ m];
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          const double dx = p[r].x - q0.x, dy = p[r].y - q0.y, dz = p[r].z - q1.x;
          const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
          const double sig2 = p[r].w + q1.y;
          const double ri = rsqrt_f64(r2);
          double qh, fh, dp;
          if (KERN == KERNEL_GAUSSIAN) {
            gauss_f64(r2, sig2, ri, qh, fh, dp);
          } else {
            const double wr = rsqrt_f64(r2 + sig2);
            const double ri2 = ri * ri;
            const double w2 = wr * wr;
            const double w4 = w2 * w2;
            const double uu = sig2 * w2;
            const double u2 = uu * uu;
            const double u4 = u2 * u2;
            dp = u4 * uu * (w4 * wr);
            const double zc = dp * sig2;
            const double ph = fma(1.5, sig2, r2) * w4 * ri;
            qh = fma(-7.5, zc, ph) * sig2 * ri2;
            fh = fma(2.5, zc, -qh) * ri2;
          }
          const double wx = fma(a[r].y, q3.x, -a[r].z * q2.y);
          const double wy = fma(a[r].z, q2.x, -a[r].x * q3.x);
          const double wz = fma(a[r].x, q2.y, -a[r].y * q2.x);
          const double ft = 3.0 * fh * fma(dz, wz, fma(dy, wy, dx * wx));
          double sx = fma(ft, dx, qh * wx), sy = fma(ft, dy, qh * wy), sz = fma(ft, dz, qh * wz);
          if (DIFF) {
            const double kd = kap * dp;
            sx = fma(kd, fma(a[r].w, q2.x, -q3.y * a[r].x), sx);
            sy = fma(kd, fma(a[r].w, q2.y, -q3.y * a[r].y), sy);
            sz = fma(kd, fma(a[r].w, q3.x, -q3.y * a[r].z), sz);
          }
          if (DIAG) {
            const bool own = m == 0 && r == self;
            qh = own ? 0.0 : qh;
            sx = own ? 0.0 : sx;
            sy = own ? 0.0 : sy;
            sz = own ? 0.0 : sz;
          }
          if (SIDE != SIDE_J) {
            sum[r].ux = fma(qh, fma(q2.y, dz, -q3.x * dy), sum[r].ux);
            sum[r].uy = fma(qh, fma(q3.x, dx, -q2.x * dz), sum[r].uy);
            sum[r].uz = fma(qh, fma(q2.x, dy, -q2.y * dx), sum[r].uz);
            sum[r].sx += sx;
            sum[r].sy += sy;
            sum[r].sz += sz;
          }
          if (!DIAG && SIDE != SIDE_I) {
            // alpha_i x d and s, taken from the source's sums at the end
            b.ux = fma(qh, fma(a[r].y, dz, -a[r].z * dy), b.ux);
            b.uy = fma(qh, fma(a[r].z, dx, -a[r].x * dz), b.uy);
            b.uz = fma(qh, fma(a[r].x, dy, -a[r].y * dx), b.uz);
            b.sx += sx;
            b.sy += sy;
            b.sz += sz;
          }
        }
        if (!DIAG && SIDE != SIDE_I) rotate(b, (m ^ (m + 1)) & 31);
      }
      if (!DIAG && SIDE != SIDE_I) add64(b, -kInv4Pi, accJ + 32 * k + lane);
      __syncwarp();
    }
    if (SIDE == SIDE_J) continue;
#pragma unroll
    for (int r = 0; r < kR; ++r) add64(sum[r], kInv4Pi, accI + t0 + 32 * r + lane);
  }
}

template <bool DIFF, int KERN>
struct Pair64 {
  static constexpr int kStageBytes = kStage64;
  template <int SIDE>
  static __device__ __forceinline__ void tile_pair(const SymSeg &sg, int I, int J, int k0, int k1, int, int, char *st,
                                                   int lane, double *accI, double *accJ) {
    if (SIDE == SIDE_BOTH && I == J)
      pairs64<SIDE_BOTH, true, DIFF, KERN>(sg, I, J, k0, k1, st, lane, accI, accJ);
    else
      pairs64<SIDE, false, DIFF, KERN>(sg, I, J, k0, k1, st, lane, accI, accJ);
  }
};

template <bool DIFF, int KERN>
__global__ void __launch_bounds__(kThreads, Shape64<KERN>::blocks)
    sym_f64_group_kernel(const SymItem *__restrict__ items, const SymSeg *segs,
                         const int *__restrict__ jbase, double *__restrict__ slots) {
  group_item<Pair64<DIFF, KERN>>(items, segs, jbase, slots);
}

template <bool DIFF, int KERN>
__global__ void __launch_bounds__(kThreads, Shape64<KERN>::blocks)
    sym_f64_tile_kernel(const SymItem *__restrict__ items, const SymSeg *segs,
                        const int *__restrict__ jbase, double *__restrict__ slots) {
  tile_item<Pair64<DIFF, KERN>>(items, segs, jbase, slots);
}

template <bool DIFF, int KERN>
__global__ void __launch_bounds__(kThreads, Shape64<KERN>::blocks)
    sym_f64_group_sided_kernel(const SymItem *__restrict__ items, const SymSeg *segs,
                               const int *__restrict__ jbase, double *__restrict__ slots) {
  sided_item<Pair64<DIFF, KERN>, true>(items, segs, jbase, slots);
}

template <bool DIFF, int KERN>
__global__ void __launch_bounds__(kThreads, Shape64<KERN>::blocks)
    sym_f64_tile_sided_kernel(const SymItem *__restrict__ items, const SymSeg *segs,
                              const int *__restrict__ jbase, double *__restrict__ slots) {
  sided_item<Pair64<DIFF, KERN>, false>(items, segs, jbase, slots);
}

template <int KERN>
SymKernel select_k(bool group, bool sided, bool diffusion) {
  if (sided && group) return diffusion ? &sym_f64_group_sided_kernel<true, KERN> : &sym_f64_group_sided_kernel<false, KERN>;
  if (sided) return diffusion ? &sym_f64_tile_sided_kernel<true, KERN> : &sym_f64_tile_sided_kernel<false, KERN>;
  if (group) return diffusion ? &sym_f64_group_kernel<true, KERN> : &sym_f64_group_kernel<false, KERN>;
  return diffusion ? &sym_f64_tile_kernel<true, KERN> : &sym_f64_tile_kernel<false, KERN>;
}

SymKernel select(bool group, bool sided, bool diffusion, int kernel) {
  return kernel == KERNEL_GAUSSIAN ? select_k<KERNEL_GAUSSIAN>(group, sided, diffusion)
                                   : select_k<KERNEL_HIGHORDER>(group, sided, diffusion);
}

}  // namespace

bool pairs_f64_supported(const PairConfig &c, int kernel) {
  return c.p == 1 && c.r == 1 && c.packed == 0 && (c.tb == 128 || c.tb == 256) &&
         (kernel == KERNEL_HIGHORDER || kernel == KERNEL_GAUSSIAN);
}

cudaError_t sym_f64_occupancy(bool diffusion, int kernel, int *blocks_per_sm) {
  return sym_occupancy(select(true, false, diffusion, kernel), sym_smem_bytes(SYM_GROUP, kStage64), blocks_per_sm);
}

cudaError_t launch_sym_f64(bool group, bool sided, bool diffusion, int kernel, const SymItem *items, int n_items, int,
                           const SymSeg *segs, const int *jbase, double *slots, cudaStream_t s) {
  return sym_launch(select(group, sided, diffusion, kernel), group ? SYM_GROUP : SYM_TILE, kStage64, items, n_items, segs,
                    jbase, slots, s);
}

}  // namespace pawan
