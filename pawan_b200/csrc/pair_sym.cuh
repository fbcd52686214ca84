// The items of the symmetric pair engine, shared by its FP32 (pair_sym.cu) and
// FP64 (pair_f64.cu) kernels: which tile pairs a block of four warps computes,
// and where its sums go.  F::tile_pair computes, in one warp, sub-blocks [k0, k1)
// of 32 sources of tile J >= I against the targets [t0, t1) of tile I (a form
// that needs all of them takes them when t0 is 0), adding to accI ([6][128], tile
// I's sums) and accJ ([6][128], tile J's); F::kStageBytes is a warp's shared
// memory.
#pragma once

#include <mutex>
#include <set>
#include <utility>

#include "device.cuh"
#include "kernels.h"

namespace pawan {
namespace {

constexpr int kWarps = 4;
constexpr int kThreads = 32 * kWarps;
constexpr int kT = kSymTile;  // particles per tile
constexpr unsigned kFull = 0xffffffffu;

// Large systems: item = group a of four tiles against the groups [b0, b1).
template <class F>
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
  for (int q = tid; q < kWarps * 6 * kT; q += kThreads) accI[q] = 0.0;
  for (int b = it.b0; b < it.b1; ++b) {
    for (int q = tid; q < kWarps * 6 * kT; q += kThreads) accJ[q] = 0.0;
    __syncthreads();
    for (int r = 0; r < kWarps; ++r) {
      const int c = (warp + r) & 3;
      const int I = it.a * kWarps + warp, J = b * kWarps + c;
      // inside one group: each unordered tile pair once (rounds 0, 1 and half of 2)
      const bool mine = b > it.a || r < 2 || (r == 2 && warp < 2);
      if (mine && I < nt && J < nt)
        F::tile_pair(sg, min(I, J), max(I, J), 0, 4, 0, kT, st, lane,
                     (I <= J ? accI + warp * 6 * kT : accJ + c * 6 * kT),
                     (I <= J ? accJ + c * 6 * kT : accI + warp * 6 * kT));
      __syncthreads();
    }
    if (b == it.a) {
      for (int q = tid; q < kWarps * 6 * kT; q += kThreads) accI[q] += accJ[q];
    } else {
      const int jb = jbase[it.jb + b];
      if (jb >= 0) {
        double *out = slots + ((size_t)jb + it.a - it.row0) * kWarps * 6 * kT;
        for (int q = tid; q < kWarps * 6 * kT; q += kThreads) out[q] = accJ[q];
      }
    }
    __syncthreads();
  }
  if (it.islot >= 0) {
    double *out = slots + (size_t)it.islot * kWarps * 6 * kT;
    for (int q = tid; q < kWarps * 6 * kT; q += kThreads) out[q] = accI[q];
  }
}

// Small systems: item = one tile pair (a, b0); each warp 32 sources of tile b0.
// HALVES = 2: eight warps, the second four taking the upper 64 targets where
// the tile pair's class visits the targets in passes of 64 (the same sums, bit
// for bit): for launches of no more blocks than SMs, which wait for one tile
// pair's chain of steps.
template <class F, int HALVES>
__device__ __forceinline__ void tile_item(const SymItem *__restrict__ items, const SymSeg *segs,
                                          const int *__restrict__ jbase, double *__restrict__ slots) {
  extern __shared__ float4 smem_sym[];
  double *const accI = reinterpret_cast<double *>(smem_sym);  // [4 sub-blocks][6][128]
  double *const accJ = accI + kWarps * 6 * kT;                // [HALVES][6][128]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int sub = warp & 3, half = HALVES == 1 ? 0 : warp >> 2;
  char *const st = reinterpret_cast<char *>(accJ + HALVES * 6 * kT) + warp * F::kStageBytes;
  const SymItem it = items[blockIdx.x];
  double *const mine = accI + sub * 6 * kT;
  start_next();
  if (HALVES == 1) {
    // each lane clears what it will add to
#pragma unroll
    for (int q = 0; q < 24; ++q) mine[32 * q + lane] = 0.0;
#pragma unroll
    for (int k = 0; k < 6; ++k) accJ[k * kT + tid] = 0.0;
  } else {
    for (int q = tid; q < (kWarps + HALVES) * 6 * kT; q += HALVES * kThreads) accI[q] = 0.0;
    __syncthreads();
  }
  const SymSeg &sg = wait_previous(segs)[it.seg];
  F::tile_pair(sg, it.a, it.b0, sub, sub + 1, half * (kT / HALVES), (half + 1) * (kT / HALVES), st, lane, mine,
               accJ + half * 6 * kT);
  const int jb = it.b0 > it.a ? jbase[it.jb + it.b0] : -1;
  if (HALVES == 1 && jb >= 0) {
    // this thread's own source
    double *out = slots + ((size_t)jb + it.a) * 6 * kT;
#pragma unroll
    for (int k = 0; k < 6; ++k) out[k * kT + tid] = accJ[k * kT + tid];
  }
  __syncthreads();
  if (HALVES == 2 && jb >= 0) {
    double *out = slots + ((size_t)jb + it.a) * 6 * kT;
#pragma unroll
    for (int k = 0; k < 6 / HALVES; ++k) {
      const int q = k * HALVES * kThreads + tid;
      out[q] = accJ[q] + accJ[6 * kT + q];
    }
  }
  if (it.islot >= 0) {
    double *out = slots + (size_t)it.islot * 6 * kT;
#pragma unroll
    for (int k = 0; k < 6 / HALVES; ++k) {
      const int q = k * HALVES * kThreads + tid;
      out[q] = ((accI[q] + accI[6 * kT + q]) + accI[12 * kT + q]) + accI[18 * kT + q];
    }
  }
}

using SymKernel = void (*)(const SymItem *, const SymSeg *, const int *, double *);

// How a launch's blocks are shaped: groups of tiles, single tile pairs, or
// single tile pairs with the targets in halves.
enum SymShape { SYM_GROUP = 0, SYM_TILE = 1, SYM_TILE_HALVES = 2 };

inline int sym_threads(int shape) { return shape == SYM_TILE_HALVES ? 2 * kThreads : kThreads; }

inline size_t sym_smem_bytes(int shape, size_t stage) {
  const size_t tile = (size_t)6 * kT * sizeof(double);
  const size_t source_sums = shape == SYM_GROUP ? kWarps : shape == SYM_TILE ? 1 : 2;
  return (kWarps + source_sums) * tile + (size_t)(sym_threads(shape) / 32) * stage;
}

// Opts a kernel in to its dynamic shared memory beyond the default 48 KB (once
// per kernel and device).
inline cudaError_t sym_prepare(SymKernel f, size_t bytes) {
  static std::mutex mu;
  static std::set<std::pair<int, SymKernel>> done;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(mu);
  if (done.count({dev, f})) return cudaSuccess;
  e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) done.insert({dev, f});
  return e;
}

inline cudaError_t sym_occupancy(SymKernel f, size_t bytes, int *blocks_per_sm) {
  cudaError_t e = sym_prepare(f, bytes);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, f, kThreads, bytes);
}

inline cudaError_t sym_launch(SymKernel f, int threads, size_t bytes, const SymItem *items, int n_items, const SymSeg *segs,
                              const int *jbase, double *slots, cudaStream_t s) {
  if (n_items <= 0) return cudaSuccess;
  cudaError_t e = sym_prepare(f, bytes);
  if (e != cudaSuccess) return e;
  return launch_dependent(f, dim3(n_items), threads, bytes, s, items, segs, jbase, slots);
}

}  // namespace
}  // namespace pawan
