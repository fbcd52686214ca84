// The items of the symmetric pair engine, shared by its FP32 (pair_sym.cu) and
// FP64 (pair_f64.cu) kernels: which tile pairs a block of four warps computes,
// and where its sums go.  F::tile_pair computes sub-blocks of 32 sources of tile
// J >= I against tile I in one warp, adding to accI ([6][128], tile I's sums)
// and accJ ([6][128], tile J's); F::kStageBytes is a warp's shared memory.
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
__device__ __forceinline__ void group_item(const SymItem *__restrict__ items, const SymSeg *__restrict__ segs,
                                           const int *__restrict__ jbase, double *__restrict__ slots) {
  extern __shared__ float4 smem_sym[];
  double *const accI = reinterpret_cast<double *>(smem_sym);  // [4 warps][6][128]
  double *const accJ = accI + kWarps * 6 * kT;                // [4 tiles][6][128]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  char *const st = reinterpret_cast<char *>(accJ + kWarps * 6 * kT) + warp * F::kStageBytes;
  const SymItem it = items[blockIdx.x];
  const SymSeg &sg = segs[it.seg];
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
        F::tile_pair(sg, min(I, J), max(I, J), 0, 4, st, lane,
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
template <class F>
__device__ __forceinline__ void tile_item(const SymItem *__restrict__ items, const SymSeg *__restrict__ segs,
                                          const int *__restrict__ jbase, double *__restrict__ slots) {
  extern __shared__ float4 smem_sym[];
  double *const accI = reinterpret_cast<double *>(smem_sym);  // [4 warps][6][128]
  double *const accJ = accI + kWarps * 6 * kT;                // [6][128]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  char *const st = reinterpret_cast<char *>(accJ + 6 * kT) + warp * F::kStageBytes;
  const SymItem it = items[blockIdx.x];
  const SymSeg &sg = segs[it.seg];
  double *const mine = accI + warp * 6 * kT;
#pragma unroll
  for (int q = 0; q < 24; ++q) mine[32 * q + lane] = 0.0;
#pragma unroll
  for (int k = 0; k < 6; ++k) accJ[k * kT + tid] = 0.0;
  F::tile_pair(sg, it.a, it.b0, warp, warp + 1, st, lane, mine, accJ);
  if (it.b0 > it.a) {
    const int jb = jbase[it.jb + it.b0];
    if (jb >= 0) {
      // this thread's own source
      double *out = slots + ((size_t)jb + it.a) * 6 * kT;
#pragma unroll
      for (int k = 0; k < 6; ++k) out[k * kT + tid] = accJ[k * kT + tid];
    }
  }
  __syncthreads();
  if (it.islot >= 0) {
    double *out = slots + (size_t)it.islot * 6 * kT;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int q = k * kT + tid;
      out[q] = ((accI[q] + accI[6 * kT + q]) + accI[12 * kT + q]) + accI[18 * kT + q];
    }
  }
}

using SymKernel = void (*)(const SymItem *, const SymSeg *, const int *, double *);

inline size_t sym_smem_bytes(bool group, size_t stage) {
  const size_t acc = (size_t)kWarps * 6 * kT * sizeof(double);
  return acc + (group ? acc : acc / kWarps) + (size_t)kWarps * stage;
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

inline cudaError_t sym_launch(SymKernel f, size_t bytes, const SymItem *items, int n_items, const SymSeg *segs,
                              const int *jbase, double *slots, cudaStream_t s) {
  if (n_items <= 0) return cudaSuccess;
  cudaError_t e = sym_prepare(f, bytes);
  if (e != cudaSuccess) return e;
  f<<<n_items, kThreads, bytes, s>>>(items, segs, jbase, slots);
  return cudaGetLastError();
}

}  // namespace
}  // namespace pawan
