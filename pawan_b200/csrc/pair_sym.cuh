// The items of the symmetric pair engine, shared by its FP32 (pair_sym.cu) and
// FP64 (pair_f64.cu) kernels: which tile pairs a block of four warps computes,
// and where its sums go.  F::tile_pair computes, in one warp, sub-blocks [k0, k1)
// of 32 sources of tile J >= I against the targets [t0, t1) of tile I (a form
// that needs all of them takes them when t0 is 0), adding to accI ([6][128], tile
// I's sums) and accJ ([6][128], tile J's), or to one of them alone (its SIDE
// parameter; those sums are the same, bit for bit); F::kStageBytes is a warp's
// shared memory.
#pragma once

#include <cooperative_groups.h>

#include "device.cuh"
#include "kernels.h"

namespace pawan {
namespace {

constexpr int kWarps = 4;
constexpr int kThreads = 32 * kWarps;
constexpr int kT = kSymTile;  // particles per tile
constexpr unsigned kFull = 0xffffffffu;

// Large systems: item = group a of four tiles against the groups [b0, b1).
template <class F, int SIDE = SIDE_BOTH>
__device__ __forceinline__ void group_item(const SymItem *__restrict__ items, const SymSeg *segs,
                                           const int *__restrict__ jbase, double *__restrict__ slots) {
  extern __shared__ float4 smem_sym[];
  double *const accI = reinterpret_cast<double *>(smem_sym);  // [4 warps][6][128]
  double *const accJ = accI + kWarps * 6 * kT;                // [4 tiles][6][128]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  char *const st = reinterpret_cast<char *>(accJ + kWarps * 6 * kT) + warp * F::kStageBytes;
  const SymItem it = items[blockIdx.x];
  start_next();
  const SymSeg &sg = wait_previous(segs)[it.seg];
  const int nt = (sg.n + kT - 1) / kT;
  if (SIDE != SIDE_J)
    for (int q = tid; q < kWarps * 6 * kT; q += kThreads) accI[q] = 0.0;
  for (int b = it.b0; b < it.b1; ++b) {
    if (SIDE != SIDE_I)
      for (int q = tid; q < kWarps * 6 * kT; q += kThreads) accJ[q] = 0.0;
    __syncthreads();
    for (int r = 0; r < kWarps; ++r) {
      const int c = (warp + r) & 3;
      const int I = it.a * kWarps + warp, J = b * kWarps + c;
      // inside one group: each unordered tile pair once (rounds 0, 1 and half of 2)
      const bool mine = b > it.a || r < 2 || (r == 2 && warp < 2);
      if (mine && I < nt && J < nt)
        F::template tile_pair<SIDE>(sg, min(I, J), max(I, J), 0, 4, 0, kT, st, lane,
                                    (I <= J ? accI + warp * 6 * kT : accJ + c * 6 * kT),
                                    (I <= J ? accJ + c * 6 * kT : accI + warp * 6 * kT));
      __syncthreads();
    }
    if (SIDE == SIDE_I) {
      continue;  // (nothing of group b is kept, and the round above ended in a barrier)
    } else if (b == it.a) {
      for (int q = tid; q < kWarps * 6 * kT; q += kThreads) accI[q] += accJ[q];
    } else {
      const int jb = jbase[it.jb + b];
      if (jb != kNoSlot) {
        double *out = slots + (size_t)(jb + it.a) * kWarps * 6 * kT;
        for (int q = tid; q < kWarps * 6 * kT; q += kThreads) out[q] = accJ[q];
      }
    }
    __syncthreads();
  }
  if (it.islot != kNoSlot) {
    double *out = slots + (size_t)it.islot * kWarps * 6 * kT;
    for (int q = tid; q < kWarps * 6 * kT; q += kThreads) out[q] = accI[q];
  }
}

// Small systems: item = one tile pair (a, b0); each warp 32 of its sources.
template <class F, int SIDE = SIDE_BOTH>
__device__ __forceinline__ void tile_item(const SymItem *__restrict__ items, const SymSeg *segs,
                                          const int *__restrict__ jbase, double *__restrict__ slots) {
  extern __shared__ float4 smem_sym[];
  double *const accI = reinterpret_cast<double *>(smem_sym);  // [4 sub-blocks][6][128]
  double *const accJ = accI + kWarps * 6 * kT;                // [6][128]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  char *const st = reinterpret_cast<char *>(accJ + 6 * kT) + warp * F::kStageBytes;
  const SymItem it = items[blockIdx.x];
  double *const mine = accI + warp * 6 * kT;
  start_next();
  // each lane clears what it will add to
#pragma unroll
  for (int q = 0; q < 24; ++q) mine[32 * q + lane] = 0.0;
#pragma unroll
  for (int k = 0; k < 6; ++k) accJ[k * kT + tid] = 0.0;
  const SymSeg &sg = wait_previous(segs)[it.seg];
  F::template tile_pair<SIDE>(sg, it.a, it.b0, warp, warp + 1, 0, kT, st, lane, mine, accJ);
  const int jb = it.b0 > it.a ? jbase[it.jb + it.b0] : kNoSlot;
  if (jb != kNoSlot) {
    // this thread's own source
    double *out = slots + (size_t)(jb + it.a) * 6 * kT;
#pragma unroll
    for (int k = 0; k < 6; ++k) out[k * kT + tid] = accJ[k * kT + tid];
  }
  __syncthreads();
  if (it.islot != kNoSlot) {
    double *out = slots + (size_t)it.islot * 6 * kT;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int q = k * kThreads + tid;
      out[q] = ((accI[q] + accI[6 * kT + q]) + accI[12 * kT + q]) + accI[18 * kT + q];
    }
  }
}

// The same sums, bit for bit, from eight warps: C blocks (a cluster) per tile
// pair, block c computing kSubs runs of 32 sources, each in two warps, the second
// taking the upper 64 targets where the tile pair's class visits the targets in
// passes of 64; the runs' target sums are added through distributed shared
// memory.  For launches that last as long as one tile pair's chain of steps.
template <int C>
struct Spread {
  static constexpr int subs = 4 / C;  // runs of 32 sources per block
  static constexpr int threads = 64 * subs;
};

template <class F, int C>
__device__ __forceinline__ void spread_item(const SymItem *__restrict__ items, const SymSeg *segs,
                                            const int *__restrict__ jbase, double *__restrict__ slots) {
  namespace cg = cooperative_groups;
  constexpr int kSubs = Spread<C>::subs, kN = Spread<C>::threads, kC = 6 * kT;
  extern __shared__ float4 smem_sym[];
  double *const accI = reinterpret_cast<double *>(smem_sym);  // [kSubs][6][128]
  double *const accJ = accI + kSubs * kC;                     // [2 halves][6][128], the block's sources used
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int half = warp / kSubs, own = warp % kSubs;  // (the warps of one half on different schedulers)
  char *const st = reinterpret_cast<char *>(accJ + 2 * kC) + warp * F::kStageBytes;
  const int rank = C > 1 ? (int)blockIdx.x % C : 0, sub = kSubs * rank + own;
  const SymItem it = items[blockIdx.x / C];
  SymSeg sg = segs[it.seg];
  start_next();
#pragma unroll
  for (int q = tid; q < (kSubs + 2) * kC; q += kN) accI[q] = 0.0;
  __syncthreads();
  wait_previous_for(sg.pos32, sg.vor32, sg.poslo, sg.vorlo, sg.pos64, sg.vor64, sg.boxes);
  F::template tile_pair<SIDE_BOTH>(sg, it.a, it.b0, sub, sub + 1, half * (kT / 2), (half + 1) * (kT / 2), st, lane,
                                   accI + own * kC, accJ + half * kC);
  if constexpr (C > 1)
    cg::this_cluster().sync();
  else
    __syncthreads();
  const int jb = it.b0 > it.a ? jbase[it.jb + it.b0] : kNoSlot;
  if (jb != kNoSlot) {
    // thread: one of the block's 32 kSubs sources, three of its six sums
    const int at = 3 * (tid / (32 * kSubs)) * kT + 32 * kSubs * rank + tid % (32 * kSubs);
    double *out = slots + (size_t)(jb + it.a) * kC;
#pragma unroll
    for (int u = 0; u < 3; ++u) out[at + u * kT] = accJ[at + u * kT] + accJ[kC + at + u * kT];
  }
  if (it.islot != kNoSlot) {
    const double *c[4];  // the runs of sources in order
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      c[k] = accI + (k % kSubs) * kC;
      if constexpr (C > 1) c[k] = cg::this_cluster().map_shared_rank(c[k], k / kSubs);
    }
    double *out = slots + (size_t)it.islot * kC;
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      const int q = rank * (kC / C) + u * kN + tid;
      out[q] = ((c[0][q] + c[1][q]) + c[2][q]) + c[3][q];
    }
  }
  if constexpr (C > 1) {
    // no block leaves while another reads its sums (which the stores above have
    // waited for; nothing else is to be ordered)
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  }
}

// Sharded systems: an item between a group of this process and one of another
// forms the own group's sums alone (28 of a far step's 37 operations and none of
// its shuffles, the sums bit for bit those of an unsharded launch).  One kernel for
// all three kinds, so that a launch has one last wave.  A rank's right-hand side on
// one B200, slowest of the ranks of 2 / 4 / 8, against forming both sides: ring pair
// at N = 131,072 8.59 / 4.63 / 2.48 ms, 10.38 / 6.18 / 3.42 (one-sided kernel, every
// ordered pair: 9.26 / 4.69 / 2.40); FP64 at 65,536 8.25 / 4.76 / 2.62, 9.15 / 5.45 /
// 3.01; Gaussian at 65,536 2.36 / 1.45 / 0.88, 2.91 / 1.81 / 1.13.
template <class F, bool GROUP>
__device__ __forceinline__ void sided_item(const SymItem *__restrict__ items, const SymSeg *segs,
                                           const int *__restrict__ jbase, double *__restrict__ slots) {
  const int side = items[blockIdx.x].side;
  if (GROUP) {
    if (side == SIDE_I)
      group_item<F, SIDE_I>(items, segs, jbase, slots);
    else if (side == SIDE_J)
      group_item<F, SIDE_J>(items, segs, jbase, slots);
    else
      group_item<F>(items, segs, jbase, slots);
  } else {
    if (side == SIDE_I)
      tile_item<F, SIDE_I>(items, segs, jbase, slots);
    else if (side == SIDE_J)
      tile_item<F, SIDE_J>(items, segs, jbase, slots);
    else
      tile_item<F>(items, segs, jbase, slots);
  }
}

using SymKernel = void (*)(const SymItem *, const SymSeg *, const int *, double *);

// How a launch's blocks are shaped: groups of tiles, single tile pairs, or
// single tile pairs over eight warps of one block or of a cluster of two.
enum SymShape { SYM_GROUP = 0, SYM_TILE = 1, SYM_WIDE = 2, SYM_SPREAD = 3 };
// (a sharded plan's kernel has the first two shapes only)

inline int sym_cluster(int shape) { return shape == SYM_SPREAD ? 2 : 1; }
inline int sym_threads(int shape) { return shape == SYM_WIDE ? Spread<1>::threads : kThreads; }

inline size_t sym_smem_bytes(int shape, size_t stage) {
  const size_t tile = (size_t)6 * kT * sizeof(double);
  const size_t sums = shape == SYM_GROUP  ? 2 * kWarps
                      : shape == SYM_TILE ? kWarps + 1
                                          : 2 + (shape == SYM_WIDE ? Spread<1>::subs : Spread<2>::subs);
  return sums * tile + (size_t)(sym_threads(shape) / 32) * stage;
}

inline cudaError_t sym_occupancy(SymKernel f, size_t bytes, int *blocks_per_sm) {
  cudaError_t e = allow_dynamic_smem((const void *)f, bytes);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, f, kThreads, bytes);
}

inline cudaError_t sym_launch(SymKernel f, int shape, size_t stage, const SymItem *items, int n_items,
                              const SymSeg *segs, const int *jbase, double *slots, cudaStream_t s) {
  if (n_items <= 0) return cudaSuccess;
  const size_t bytes = sym_smem_bytes(shape, stage);
  cudaError_t e = allow_dynamic_smem((const void *)f, bytes);
  if (e != cudaSuccess) return e;
  const int cluster = sym_cluster(shape);
  return launch_dependent_clusters(f, cluster, dim3(n_items * cluster), sym_threads(shape), bytes, s, items, segs,
                                   jbase, slots);
}

}  // namespace
}  // namespace pawan
