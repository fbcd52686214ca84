// Conserved / monitored quantities of a system, all in FP64.
//
// Reference (src/interaction/interaction.cpp):
//   total vorticity  sum alpha                       :240-246
//   linear impulse   1/2 sum x x alpha               :248-259
//   angular impulse  1/3 sum x x (x x alpha)         :261-275
//   enstrophy        sum_i 5/(4 pi s_i^3)|alpha_i|^2 + sum_{i != j} [F1 (a_i.a_j)
//                    + F2 (a_i.x_ij)(a_j.x_ij)]      :277-315, ENSTROPHY
//                    (interaction_utils.h:107-156), ENST (highorder.h:69-86)
//   helicity         sum_{i != j} q(rho,sigma) x_ij.(a_i x a_j)     :317-349,
//                    HELICITY (interaction_utils.h:167-190)
//   kinetic energy   2 sum_i |a_i|^2/(8 pi s_i) + sum_{i != j} w_ij KE_ij with
//                    w_ij = 2 inside a wake, 1 across wakes      :351-383,
//                    KINETICENERGY (interaction_utils.h:197-240)
// With the Gaussian kernel (src/interaction/gaussian.h) the enstrophy terms
// are the reference's stub ENST = 0 (gaussian.h:67-86) and helicity uses the
// Gaussian QSIG (:30-38): q = (phi/rho_bar - Z)/rho_bar^2 with
// phi = erf(rho_bar/sqrt 2)/(4 pi sigma^3), Z = exp(-rho_bar^2/2)/(sigma^3 (2 pi)^1.5).
// The reference's pair loops visit i<j and double (or, across wakes, double
// the full cross sum); the terms are symmetric in (i, j), so each unordered pair
// is visited once here too.  Per-target sums are reduced per block in a fixed
// tree and the block partials by one block in fixed order: deterministic.
//
// The quadratic kernel is bound by the FP64 pipe: 68 operations per unordered
// pair.  A block takes 128 targets and a range of the sources from the targets'
// own tile on, in ranges short enough that the device is full from about two
// thousand particles on.  Helical wake, whole call on one B200: N = 65,536
// 10.3 ms (28.7 when every ordered pair was visited, by one block per 128
// targets), 0.76 of the FP64 pipe's rate; N = 16,384 0.67 ms (3.2).
#include <algorithm>

#include "device.cuh"
#include "kernels.h"
#include "rsqrt64.cuh"

namespace pawan {
namespace {

constexpr int kDiagThreads = 128;
constexpr int kLin = 9;   // linear quantities
constexpr int kQuad = 3;  // enstrophy, helicity, kinetic energy
constexpr int kFinalThreads = 512;
constexpr double kDiagBlocks = 3000.0;  // five per resident block: the last ones end together

template <int K>
__device__ void block_sum(double (&v)[K], double *smem /* [K][kDiagThreads] */, double *out) {
  const int t = threadIdx.x;
#pragma unroll
  for (int k = 0; k < K; ++k) smem[k * kDiagThreads + t] = v[k];
  __syncthreads();
  for (int s = kDiagThreads / 2; s > 0; s >>= 1) {
    if (t < s) {
#pragma unroll
      for (int k = 0; k < K; ++k) smem[k * kDiagThreads + t] += smem[k * kDiagThreads + t + s];
    }
    __syncthreads();
  }
  if (t == 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) out[k] = smem[k * kDiagThreads];
  }
}

__global__ void __launch_bounds__(kDiagThreads)
    diag_linear_kernel(int n, const double4 *__restrict__ pos, const double4 *__restrict__ vor,
                       double *__restrict__ block_out) {
  __shared__ double smem[kLin * kDiagThreads];
  const int i = blockIdx.x * kDiagThreads + threadIdx.x;
  double v[kLin];
#pragma unroll
  for (int k = 0; k < kLin; ++k) v[k] = 0.0;
  if (i < n) {
    const double4 r = pos[i], a = vor[i];
    const double rxa0 = r.y * a.z - r.z * a.y;
    const double rxa1 = r.z * a.x - r.x * a.z;
    const double rxa2 = r.x * a.y - r.y * a.x;
    v[0] = a.x;
    v[1] = a.y;
    v[2] = a.z;
    v[3] = rxa0;
    v[4] = rxa1;
    v[5] = rxa2;
    v[6] = r.y * rxa2 - r.z * rxa1;
    v[7] = r.z * rxa0 - r.x * rxa2;
    v[8] = r.x * rxa1 - r.y * rxa0;
  }
  block_sum<kLin>(v, smem, block_out + (size_t)blockIdx.x * kLin);
}

// Block (c, I): targets of tile I against the sources j > i of
// [128 I + c * span, 128 I + (c + 1) * span).
template <int KERN>
__global__ void __launch_bounds__(kDiagThreads)
    diag_quadratic_kernel(int n, int tile0, int span, const double4 *__restrict__ pos, const double4 *__restrict__ vor,
                          const int *__restrict__ wake_id, double *__restrict__ block_out) {
  __shared__ double4 sp[kDiagThreads];  // w: s^2 / 2
  __shared__ double4 sv[kDiagThreads];
  __shared__ int sw[kDiagThreads];
  __shared__ double smem[kQuad * kDiagThreads];
  const int tid = threadIdx.x;
  const int I = tile0 + blockIdx.y;
  const int i = I * kDiagThreads + tid;
  double *const out = block_out + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * kQuad;
  const long long first = (long long)I * kDiagThreads + (long long)blockIdx.x * span;
  if (first >= n) {
    if (tid < kQuad) out[tid] = 0.0;
    return;
  }
  const int s0 = (int)first, s1 = (int)min((long long)n, first + span);
  const bool valid = i < n;
  double4 ri = make_double4(0, 0, 0, 1), ai = make_double4(0, 0, 0, 0);
  int wi = -1;
  if (valid) {
    ri = pos[i];
    ai = vor[i];
    wi = wake_id[i];
  }
  const double hi = 0.5 * ri.w * ri.w;
  double ens = 0.0, hel = 0.0, all = 0.0, same = 0.0;
  for (int ts = s0; ts < s1; ts += kDiagThreads) {
    __syncthreads();
    const int j = ts + tid;
    if (j < s1) {
      const double4 r = pos[j];
      sp[tid] = make_double4(r.x, r.y, r.z, 0.5 * r.w * r.w);
      sv[tid] = vor[j];
      sw[tid] = wake_id[j];
    }
    __syncthreads();
    const int cnt = min(kDiagThreads, s1 - ts);
    const int own = i - ts;  // sources up to the target itself belong to the other order
#pragma unroll 1  // (two: 10.45 ms, eight: 10.29)
    for (int jj = 0; jj < cnt; ++jj) {
      if (jj <= own) continue;
      const double4 rj = sp[jj], aj = sv[jj];
      const double x0 = rj.x - ri.x, x1 = rj.y - ri.y, x2 = rj.z - ri.z;
      const double rho2 = fma(x2, x2, fma(x1, x1, x0 * x0));
      const double sig2 = hi + rj.w;
      const double s = rho2 + sig2;
      const double w = rsqrt_f64(s), w2 = w * w, w3 = w2 * w, w4 = w2 * w2;
      const double aa = fma(ai.z, aj.z, fma(ai.y, aj.y, ai.x * aj.x));
      const double pp = fma(ai.z, x2, fma(ai.y, x1, ai.x * x0)) * fma(aj.z, x2, fma(aj.y, x1, aj.x * x0));
      const double rinv = rsqrt_f64(rho2);
      double q;
      if (KERN == KERNEL_GAUSSIAN) {
        // QSIG, gaussian.h:30-38, in units of 1 / (4 pi)
        const double sig = sqrt(sig2);
        const double rho_bar = rho2 * rinv / sig;
        const double z = kSqrt2OverPi * exp(-0.5 * rho_bar * rho_bar);
        q = (erf(kSqrtHalf * rho_bar) / rho_bar - z) / (rho_bar * rho_bar * sig2 * sig);
      } else {
        // ENST in units of 1 / (8 pi): (rho^2 + sigma^2)^(-7/2) [F1 (a_i.a_j) - 15 rho^2 (a_i.x)(a_j.x)],
        // F1 = 10 sigma^4 - 2 rho^4 - 7 sigma^2 rho^2 = 3 sigma^2 (4 sigma^2 - rho^2) - 2 (rho^2 + sigma^2)^2
        const double f1 = fma(-2.0 * s, s, 3.0 * sig2 * fma(4.0, sig2, -rho2));
        ens = fma(w4 * w3, fma(-15.0 * rho2, pp, f1 * aa), ens);
        // QSIG in units of 1 / (4 pi): q = (phi/rho_bar - Z)/rho_bar^2
        const double uu = sig2 * w2, u2 = uu * uu;
        const double zc = u2 * u2 * u2 * w3;
        const double ph = fma(1.5, sig2, rho2) * w4 * rinv;
        q = fma(-7.5, zc, ph) * sig2 * (rinv * rinv);
      }
      const double c0 = fma(ai.y, aj.z, -ai.z * aj.y);
      const double c1 = fma(ai.z, aj.x, -ai.x * aj.z);
      const double c2 = fma(ai.x, aj.y, -ai.y * aj.x);
      hel = fma(q, fma(x2, c2, fma(x1, c1, x0 * c0)), hel);
      // KINETICENERGY in units of 1 / (16 pi), counted once more inside a wake
      const double e = fma(s + sig2, aa, pp) * w3;
      all += e;
      same += sw[jj] == wi ? e : 0.0;
    }
  }
  double v[kQuad] = {0.0, 0.0, 0.0};
  if (valid) {
    v[0] = 2.0 * (kInvPi / 8.0) * ens;
    v[1] = 2.0 * kInv4Pi * hel;
    v[2] = 2.0 * (kInvPi / 16.0) * (all + same);
    if (blockIdx.x == 0) {
      const double a2 = ai.x * ai.x + ai.y * ai.y + ai.z * ai.z;
      if (KERN == KERNEL_HIGHORDER) v[0] += 5.0 * kInvPi / 4.0 / (ri.w * ri.w * ri.w) * a2;
      v[2] += 2.0 * (kInvPi * a2 / ri.w / 8.0);
    }
  }
  __syncthreads();
  block_sum<kQuad>(v, smem, out);
}

// Block 0 sums the linear rows, block 1 the quadratic ones, in a fixed order.
__global__ void __launch_bounds__(kFinalThreads)
    diag_final_kernel(int lin_rows, const double *__restrict__ lin, int quad_rows,
                      const double *__restrict__ quad, double *__restrict__ out) {
  __shared__ double part[kLin][kFinalThreads / 32];
  const bool linear = blockIdx.x == 0;
  const int rows = linear ? lin_rows : quad_rows, width = linear ? kLin : kQuad;
  const double *src = linear ? lin : quad;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int k = 0; k < width; ++k) {
    double v = 0.0;
#pragma unroll 4
    for (int b = threadIdx.x; b < rows; b += kFinalThreads) v += src[(size_t)b * width + k];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) part[k][warp] = v;
  }
  __syncthreads();
  if (threadIdx.x < width) {
    const int k = threadIdx.x;
    double v = 0.0;
    for (int w = 0; w < kFinalThreads / 32; ++w) v += part[k][w];
    if (linear)
      out[k] = k < 3 ? v : k < 6 ? v * 0.5 : v * (1.0 / 3.0);
    else
      out[kLin + k] = v;
  }
}

// Sources per block of the quadratic kernel: whole warps' worth, such that
// about kDiagBlocks blocks are not empty (half of the grid is).
int diag_span(int n) {
  const double tiles = (double)((n + kDiagThreads - 1) / kDiagThreads);
  const double per = std::min((double)n, 0.5 * tiles * (double)n / kDiagBlocks);
  return 32 * std::max(1, (int)(per / 32.0));
}

int diag_chunks(int n) {
  const int span = diag_span(n);
  return (n + span - 1) / span;
}

}  // namespace

size_t diag_scratch_doubles(int n) {
  const size_t nblk = (size_t)(n + kDiagThreads - 1) / kDiagThreads;
  return nblk * (kLin + (size_t)diag_chunks(n) * kQuad);
}

cudaError_t launch_diagnostics(int n, int kernel, const double4 *pos64, const double4 *vor64,
                               const int *wake_id, double *scratch, double *out, bool quadratic,
                               cudaStream_t s) {
  if (n <= 0) return cudaErrorInvalidValue;
  const int nblk = (n + kDiagThreads - 1) / kDiagThreads;
  double *lin = scratch;
  double *quad = scratch + (size_t)nblk * kLin;
  diag_linear_kernel<<<nblk, kDiagThreads, 0, s>>>(n, pos64, vor64, lin);
  const int span = diag_span(n), chunks = diag_chunks(n);
  // tiles in y in slices of the grid's extent (65,535)
  for (int t0 = 0; quadratic && t0 < nblk; t0 += 65535) {
    const dim3 grid(chunks, std::min(65535, nblk - t0));
    double *q = quad + (size_t)t0 * chunks * kQuad;
    if (kernel == KERNEL_GAUSSIAN)
      diag_quadratic_kernel<KERNEL_GAUSSIAN><<<grid, kDiagThreads, 0, s>>>(n, t0, span, pos64, vor64, wake_id, q);
    else
      diag_quadratic_kernel<KERNEL_HIGHORDER><<<grid, kDiagThreads, 0, s>>>(n, t0, span, pos64, vor64, wake_id, q);
  }
  diag_final_kernel<<<quadratic ? 2 : 1, kFinalThreads, 0, s>>>(nblk, lin, nblk * chunks, quad, out);
  return cudaGetLastError();
}

}  // namespace pawan
