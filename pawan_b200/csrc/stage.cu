// Per-particle stage kernel: reads the rates (u | dalpha) the pair kernel
// summed, applies the RK4 stage update in FP64 with the reference's operation
// order, packs the new state into the FP32 hi/lo and FP64 tile arrays the next
// pair launch reads, and writes the bounding box of each source tile.  One
// thread per particle, HBM-bound.
//
// Reference: __rk4::step (src/integration/rk4.cpp:12-76):
//   x1 = k1*(0.5 dt) + x        (:29-31)      STAGE_K1
//   x2 = k2*(0.5 dt) + x        (:39-41)      STAGE_K2
//   x3 = k3*dt + x              (:49-51)      STAGE_K3 (also forms k2 + k3, :61)
//   x += (k1 + k4)*(dt/6) + (k2 + k3)*(dt/3)   (:58-66)   STAGE_FINAL
// and __integration::step (src/integration/integration.cpp:37-45): x += r*dt.
// For a system sharded over processes, STAGE_SHARD writes this process's
// block of reduced rates to the exchange buffer, and after the all-gather the
// stage modes read every particle's rates from the gathered buffer.
// Products and sums use __dmul_rn/__dadd_rn so no multiply-add is contracted,
// keeping the update bit-identical to the reference's for equal rates.
#include <cuda_pipeline.h>

#include "device.cuh"
#include "kernels.h"

namespace pawan {
namespace {

// Blocks per SM the register budget is held to: a segment of 131,072
// particles is 512 blocks of 256, one wave at four blocks per SM on 148 SMs.
// The descriptor is read through a reference (uniform, L1-cached) rather than
// copied, which is what frees the registers.
constexpr int kStageMinBlocks = 4;

// Packs one particle: FP32 hi/lo pairs of the position relative to the
// system's origin and of the strength, plus the FP64 copies.  Returns the hi
// position and h = s^2/2 for the tile's bounding box.
__device__ __forceinline__ float4 pack(const StageDesc &d, int l, const double x[6]) {
  const double s = d.rad[l];
  const double v = d.vol[l];
  const double rx = x[0] - d.ox, ry = x[1] - d.oy, rz = x[2] - d.oz;
  const float hx = (float)rx, hy = (float)ry, hz = (float)rz;
  const float ax = (float)x[3], ay = (float)x[4], az = (float)x[5];
  const float hw = (float)(0.5 * s * s);
  d.pos32[l] = make_float4(hx, hy, hz, hw);
  d.poslo[l] = make_float4((float)(rx - (double)hx), (float)(ry - (double)hy),
                           (float)(rz - (double)hz), 0.f);
  d.vor32[l] = make_float4(ax, ay, az, (float)v);
  d.vorlo[l] = make_float4((float)(x[3] - (double)ax), (float)(x[4] - (double)ay),
                           (float)(x[5] - (double)az), 0.f);
  d.pos64[l] = make_double4(x[0], x[1], x[2], s);
  d.vor64[l] = make_double4(x[3], x[4], x[5], v);
  return make_float4(hx, hy, hz, hw);
}

// A warp's bounding box into column `warp` of wv: lower bounds of (x, y, z, h) in
// rows 0..3, upper bounds in rows 4..7; lanes without a particle contribute
// nothing.
template <int WARPS>
__device__ __forceinline__ void warp_box(float4 p, bool has, int lane, int warp, float (*wv)[WARPS]) {
  float v[8] = {has ? p.x : INFINITY,  has ? p.y : INFINITY,  has ? p.z : INFINITY,
                has ? p.w : INFINITY,  has ? p.x : -INFINITY, has ? p.y : -INFINITY,
                has ? p.z : -INFINITY, has ? p.w : -INFINITY};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = fminf(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
      v[4 + k] = fmaxf(v[4 + k], __shfl_xor_sync(0xffffffffu, v[4 + k], o));
    }
  }
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < 8; ++k) wv[k][warp] = v[k];
  }
}

// Bounding boxes of the block's tiles (box_tile particles each, aligned to
// the segment); particles beyond n contribute nothing.  The box's w components
// carry the tile's smallest (lo) and largest (hi) h = s^2/2, so the pair
// kernel can tell tile pairs of one smoothing radius.  Each warp reduces its
// 32 particles by shuffles, then one thread per tile combines the tile's
// warps (4 or 8) from shared memory: one barrier.
__device__ __forceinline__ void tile_boxes(const StageDesc &d, int l0, float4 p, bool has) {
  constexpr int kWarps = kStageThreads / 32;
  __shared__ float wv[8][kWarps];
  const int t = threadIdx.x;
  warp_box(p, has, t & 31, t >> 5, wv);
  __syncthreads();
  const int wpt = d.box_tile / 32;
  if (t < kStageThreads / d.box_tile && l0 + t * d.box_tile < d.n) {
    float lo[4], hi[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      lo[k] = wv[k][t * wpt];
      hi[k] = wv[4 + k][t * wpt];
    }
    for (int w = 1; w < wpt; ++w) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        lo[k] = fminf(lo[k], wv[k][t * wpt + w]);
        hi[k] = fmaxf(hi[k], wv[4 + k][t * wpt + w]);
      }
    }
    const int b = (l0 + t * d.box_tile) / d.box_tile;
    d.boxes[2 * b] = make_float4(lo[0], lo[1], lo[2], lo[3]);
    d.boxes[2 * b + 1] = make_float4(hi[0], hi[1], hi[2], hi[3]);
  }
}

template <int MODE>
__global__ void __launch_bounds__(kStageThreads, kStageMinBlocks)
    stage_kernel(const StageItem *__restrict__ items, const StageDesc *__restrict__ descs) {
  const StageItem it = items[blockIdx.x];
  const StageDesc &d = descs[it.seg];
  const int l = it.l0 + threadIdx.x;
  const bool has = l < d.n;
  const size_t n = (size_t)d.n;
  size_t idx[6];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    idx[k] = 3 * (size_t)l + k;
    idx[3 + k] = 3 * n + 3 * (size_t)l + k;
  }

  double r[6] = {0, 0, 0, 0, 0, 0};
  if (MODE != STAGE_PACK && has) {
    if (MODE != STAGE_SHARD && d.xchg_in) {
      const size_t S = (size_t)d.shard;
      const double *g = d.xchg_in + ((size_t)l / S) * 6 * S + (size_t)l % S;
#pragma unroll
      for (int k = 0; k < 6; ++k) r[k] = g[(size_t)k * S];
    } else {
      // the pair kernel's rates (its chunks already summed); read once, so
      // streaming loads keep them from evicting the state from L2
#pragma unroll
      for (int k = 0; k < 6; ++k) r[k] = __ldcs(d.rates + (size_t)k * n + l);
    }
  }
  if (MODE == STAGE_SHARD) {
    if (has) {
      double *o = d.xchg_out + (l - d.shard_first);
#pragma unroll
      for (int k = 0; k < 6; ++k) o[(size_t)k * d.shard] = r[k];
    }
    return;
  }

  // Per-segment step size; the coefficients are formed as the reference forms
  // them (0.5*dt, dt/6., dt/3.), and device division is correctly rounded.
  const double dt = d.dt;
  const double half = 0.5 * dt;
  const double full = dt;
  const double sixth = dt / 6.;
  const double third = dt / 3.;

  if (MODE == STAGE_RATES) {
    if (has) {
#pragma unroll
      for (int k = 0; k < 6; ++k) d.R[idx[k]] = r[k];
    }
    return;  // uniform across the block: no pack, no boxes
  }
  double x[6] = {0, 0, 0, 0, 0, 0};
  if (has) {
    if (MODE == STAGE_K1 || MODE == STAGE_K2) {
      double *K = (MODE == STAGE_K1) ? d.K1 : d.K2;
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        K[idx[k]] = r[k];
        x[k] = __dadd_rn(__dmul_rn(r[k], half), d.X[idx[k]]);
        d.Xs[idx[k]] = x[k];
      }
    } else if (MODE == STAGE_K3) {
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        d.K2[idx[k]] = __dadd_rn(d.K2[idx[k]], r[k]);
        x[k] = __dadd_rn(__dmul_rn(r[k], full), d.X[idx[k]]);
        d.Xs[idx[k]] = x[k];
      }
    } else if (MODE == STAGE_FINAL) {
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const double a = __dmul_rn(__dadd_rn(d.K1[idx[k]], r[k]), sixth);
        const double b = __dmul_rn(d.K2[idx[k]], third);
        x[k] = __dadd_rn(d.X[idx[k]], __dadd_rn(a, b));
        d.X[idx[k]] = x[k];
      }
    } else if (MODE == STAGE_EULER) {
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        x[k] = __dadd_rn(d.X[idx[k]], __dmul_rn(r[k], full));
        d.X[idx[k]] = x[k];
      }
    } else {  // STAGE_PACK
#pragma unroll
      for (int k = 0; k < 6; ++k) x[k] = d.X[idx[k]];
    }
  }
  float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
  if (has) p = pack(d, l, x);
  tile_boxes(d, it.l0, p, has);
}

// The stage update of a plan on the symmetric engine whose slots are all written
// by one wave: one block per 128-particle tile sums the tile's slots (four
// threads per particle, a quarter of the slots each, the quarters then in
// order), updates the 768 state components one per thread -- contiguous in
// the state vectors, where one thread per particle strides by three -- and
// packs the tile.  In place of a launch for the sums and one for the stage: a
// right-hand side at N = 2,048 20.6 us against 24.6, at 512 20.6 against 24.6
// (eager RK4 on one B200, before launches overlapped).
//
// What bounds it: the latency of its chain of loads (small systems) and the L2's
// bytes in flight (a tile of N = 16,384 has 128 slots of 6 KB).  The state is
// loaded beside the slots, by copies to shared memory that hold no registers,
// and the registers are left unbounded (some 95): more slot loads in flight, and
// one block to an SM -- with 40 registers the blocks, which start while the pair
// kernel's last ones run, gather three to an SM on the SMs that are free first.
// One RK4 right-hand side, 40 registers / unbounded: N = 2,048 17.3 / 14.7 us,
// 8,192 84.0 / 79.2, 16,384 285 / 265.  (8-byte copies of the slots to shared
// memory, three or four slots deep: 18.1, 88.2, 283.)
constexpr int kSumThreads = 4 * kSymTile;

// A block's quarter sums of a tile's slots: part[quarter][component][particle].
__device__ __forceinline__ void sum_slots(const SymSum &s, const double *slots, double (*part)[6][kSymTile]) {
  const int q = threadIdx.x & (kSymTile - 1), g = threadIdx.x / kSymTile;
  const int c0 = s.count * g / 4, c1 = s.count * (g + 1) / 4;
  double a[6] = {0, 0, 0, 0, 0, 0};
  const double *p = slots + s.first + q;
#pragma unroll 4
  for (int c = c0; c < c1; ++c) {
#pragma unroll
    for (int k = 0; k < 6; ++k) a[k] += __ldcs(p + (size_t)c * s.stride + k * kSymTile);
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) part[g][k][q] = a[k];
  __syncthreads();
}

__device__ __forceinline__ double slot_sum(const double (*part)[6][kSymTile], int k, int i) {
  return __dadd_rn(__dadd_rn(__dadd_rn(part[0][k][i], part[1][k][i]), part[2][k][i]), part[3][k][i]);
}

// The sums alone, into rates[.][128 t ..] (added to what is there when `add`):
// sharded systems, whose rates are exchanged, and plans of several waves.
__global__ void __launch_bounds__(kSumThreads, 1)
    sum_slots_kernel(const SymSum *__restrict__ sums, const StageDesc *descs, const double *slots) {
  __shared__ double part[4][6][kSymTile];
  const SymSum s = sums[blockIdx.x];
  start_next();
  slots = wait_previous(slots);
  const StageDesc &d = wait_previous(descs)[s.seg];
  sum_slots(s, slots, part);
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int e = threadIdx.x + u * kSumThreads, k = e / kSymTile, i = e % kSymTile;
    if (k >= 6 || s.t * kSymTile + i >= d.n) continue;
    double *out = const_cast<double *>(d.rates) + (size_t)k * d.n + s.t * kSymTile + i;
    const double r = slot_sum(part, k, i);
    *out = s.add ? __dadd_rn(*out, r) : r;
  }
}

template <int MODE>
__global__ void __launch_bounds__(kSumThreads, 1)
    sum_stage_kernel(const SymSum *__restrict__ sums, const StageDesc *descs, const double *slots) {
  constexpr int kT = kSymTile, kC = 6 * kSymTile;
  constexpr bool kOne = MODE == STAGE_FINAL, kTwo = MODE == STAGE_FINAL || MODE == STAGE_K3;
  __shared__ double part[4][6][kT];
  __shared__ double xs[kC];  // the state, then the new one: [x (128 x 3) | alpha (128 x 3)]
  __shared__ double k1[kOne ? kC : 1], k2[kTwo ? kC : 1];
  __shared__ float box[8][kT / 32];
  const SymSum s = sums[blockIdx.x];
  const StageDesc *const desc = descs + s.seg;
  const int n = desc->n;
  const double *X = desc->X, *K1 = desc->K1, *K2 = desc->K2;
  start_next();
  wait_previous_for(slots, X, K1, K2);
  const int tid = threadIdx.x, q = tid & (kT - 1), g = tid / kT;
  const int l0 = s.t * kT;
  // the values the update starts from, in flight beside the slots and held by no register
  if (MODE != STAGE_RATES) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int e = tid + u * kSumThreads;
      const int h = e >= kC / 2 ? 1 : 0, f = e - h * (kC / 2);  // x or alpha, component within it
      if (e >= kC || l0 + f / 3 >= n) continue;
      const size_t at = (size_t)h * 3 * n + 3 * (size_t)l0 + f;
      __pipeline_memcpy_async(xs + e, X + at, sizeof(double));
      if (kOne) __pipeline_memcpy_async(k1 + e, K1 + at, sizeof(double));
      if (kTwo) __pipeline_memcpy_async(k2 + e, K2 + at, sizeof(double));
    }
    __pipeline_commit();
  }
  sum_slots(s, slots, part);
  if (MODE != STAGE_RATES) __pipeline_wait_prior(0);  // (each thread reads its own copies)
  const StageDesc &d = *launder_pointer(desc);
  const double dt = d.dt;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int e = tid + u * kSumThreads;
    if (e >= kC) break;
    const int h = e >= kC / 2 ? 1 : 0, f = e - h * (kC / 2);
    const int i = f / 3;
    if (l0 + i >= n) continue;
    const size_t at = (size_t)h * 3 * n + 3 * (size_t)l0 + f;
    const double r = slot_sum(part, 3 * h + (f - 3 * i), i);
    double x = 0.0;
    if (MODE == STAGE_RATES) {
      d.R[at] = r;
      continue;
    }
    if (MODE == STAGE_K1 || MODE == STAGE_K2) {
      (MODE == STAGE_K1 ? d.K1 : d.K2)[at] = r;
      x = __dadd_rn(__dmul_rn(r, 0.5 * dt), xs[e]);
      d.Xs[at] = x;
    } else if (MODE == STAGE_K3) {
      d.K2[at] = __dadd_rn(k2[e], r);
      x = __dadd_rn(__dmul_rn(r, dt), xs[e]);
      d.Xs[at] = x;
    } else if (MODE == STAGE_FINAL) {
      const double a = __dmul_rn(__dadd_rn(k1[e], r), dt / 6.);
      const double b = __dmul_rn(k2[e], dt / 3.);
      x = __dadd_rn(xs[e], __dadd_rn(a, b));
      d.X[at] = x;
    } else {  // STAGE_EULER
      x = __dadd_rn(xs[e], __dmul_rn(r, dt));
      d.X[at] = x;
    }
    xs[e] = x;
  }
  if (MODE == STAGE_RATES) return;
  __syncthreads();
  // pack: each quarter of the block writes one pair of arrays
  const int l = l0 + q;
  const bool has = l < n;
  const double x0 = xs[3 * q], x1 = xs[3 * q + 1], x2 = xs[3 * q + 2];
  const double a0 = xs[kC / 2 + 3 * q], a1 = xs[kC / 2 + 3 * q + 1], a2 = xs[kC / 2 + 3 * q + 2];
  if (g == 0) {
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    if (has) {
      const double sr = d.rad[l];
      const double rx = x0 - d.ox, ry = x1 - d.oy, rz = x2 - d.oz;
      p = make_float4((float)rx, (float)ry, (float)rz, (float)(0.5 * sr * sr));
      d.pos32[l] = p;
      d.poslo[l] = make_float4((float)(rx - (double)p.x), (float)(ry - (double)p.y), (float)(rz - (double)p.z), 0.f);
    }
    warp_box(p, has, tid & 31, tid >> 5, box);
  } else if (has && g == 1) {
    const float ax = (float)a0, ay = (float)a1, az = (float)a2;
    d.vor32[l] = make_float4(ax, ay, az, (float)d.vol[l]);
    d.vorlo[l] = make_float4((float)(a0 - (double)ax), (float)(a1 - (double)ay), (float)(a2 - (double)az), 0.f);
  } else if (has && g == 2) {
    d.pos64[l] = make_double4(x0, x1, x2, d.rad[l]);
  } else if (has) {
    d.vor64[l] = make_double4(a0, a1, a2, d.vol[l]);
  }
  __syncthreads();
  if (tid < 8) {
    float v = box[tid][0];
    for (int w = 1; w < kT / 32; ++w) v = tid < 4 ? fminf(v, box[tid][w]) : fmaxf(v, box[tid][w]);
    reinterpret_cast<float *>(d.boxes + 2 * s.t)[tid] = v;
  }
}

}  // namespace

cudaError_t launch_sym_sums(const SymSum *sums, int n_sums, const StageDesc *descs, const double *slots,
                            cudaStream_t s) {
  if (n_sums <= 0) return cudaSuccess;
  return launch_dependent(sum_slots_kernel, dim3(n_sums), kSumThreads, 0, s, sums, descs, slots);
}

cudaError_t launch_sum_stage(int mode, int n_sums, const SymSum *sums, const StageDesc *descs,
                             const double *slots, cudaStream_t s) {
  if (n_sums <= 0) return cudaSuccess;
  switch (mode) {
    case STAGE_RATES:
      return launch_dependent(sum_stage_kernel<STAGE_RATES>, dim3(n_sums), kSumThreads, 0, s, sums, descs, slots);
    case STAGE_K1:
      return launch_dependent(sum_stage_kernel<STAGE_K1>, dim3(n_sums), kSumThreads, 0, s, sums, descs, slots);
    case STAGE_K2:
      return launch_dependent(sum_stage_kernel<STAGE_K2>, dim3(n_sums), kSumThreads, 0, s, sums, descs, slots);
    case STAGE_K3:
      return launch_dependent(sum_stage_kernel<STAGE_K3>, dim3(n_sums), kSumThreads, 0, s, sums, descs, slots);
    case STAGE_FINAL:
      return launch_dependent(sum_stage_kernel<STAGE_FINAL>, dim3(n_sums), kSumThreads, 0, s, sums, descs, slots);
    case STAGE_EULER:
      return launch_dependent(sum_stage_kernel<STAGE_EULER>, dim3(n_sums), kSumThreads, 0, s, sums, descs, slots);
    default:
      return cudaErrorInvalidValue;
  }
}

cudaError_t launch_stage(int mode, int n_blocks, const StageItem *items, const StageDesc *descs,
                         cudaStream_t s) {
  if (n_blocks <= 0) return cudaSuccess;
  dim3 grid(n_blocks), block(kStageThreads);
  switch (mode) {
    case STAGE_RATES:
      stage_kernel<STAGE_RATES><<<grid, block, 0, s>>>(items, descs);
      break;
    case STAGE_K1:
      stage_kernel<STAGE_K1><<<grid, block, 0, s>>>(items, descs);
      break;
    case STAGE_K2:
      stage_kernel<STAGE_K2><<<grid, block, 0, s>>>(items, descs);
      break;
    case STAGE_K3:
      stage_kernel<STAGE_K3><<<grid, block, 0, s>>>(items, descs);
      break;
    case STAGE_FINAL:
      stage_kernel<STAGE_FINAL><<<grid, block, 0, s>>>(items, descs);
      break;
    case STAGE_EULER:
      stage_kernel<STAGE_EULER><<<grid, block, 0, s>>>(items, descs);
      break;
    case STAGE_PACK:
      stage_kernel<STAGE_PACK><<<grid, block, 0, s>>>(items, descs);
      break;
    case STAGE_SHARD:
      stage_kernel<STAGE_SHARD><<<grid, block, 0, s>>>(items, descs);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace pawan
