// Host-side launchers of the pawan B200 kernels (implemented in the .cu files).
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <set>
#include <utility>

#include "device.cuh"

namespace pawan {

// Tiling of the all-pairs kernels: `tb` threads per block (= sources per
// shared-memory tile), `p` threads per target, `r` targets per thread
// (targets per block = tb / p * r), `unroll` = unroll depth of the source loop,
// `minb` = blocks per SM the registers are bounded for (0: the default),
// `packed` > 0: the symmetric engine (pair_sym.cu), which the other fields and
// `split` do not change; 0: the one-sided scalar kernel.
struct PairConfig {
  int tb;
  int p;
  int unroll;
  int r = 1;
  int minb = 0;
  int packed = 0;
  int split = 0;
  bool onesided = false;  // {128, 1, 4, 1, 0, 2} on the one-sided packed kernel
};

// Opts a kernel in to its dynamic shared memory beyond the default 48 KB (once
// per kernel and device).
inline cudaError_t allow_dynamic_smem(const void *f, size_t bytes) {
  static std::mutex mu;
  static std::set<std::pair<int, const void *>> done;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(mu);
  if (done.count({dev, f})) return cudaSuccess;
  e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) done.insert({dev, f});
  return e;
}

// Launches f on s as a programmatic dependent of the kernel before it (its
// launch overlaps that kernel's end; see wait_previous in device.cuh), in
// clusters of `cluster` blocks.
template <class... P, class... A>
inline cudaError_t launch_dependent_clusters(void (*f)(P...), int cluster, dim3 grid, int threads, size_t smem,
                                             cudaStream_t s, A... args) {
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = (unsigned)cluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = at;
  c.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&c, f, static_cast<P>(args)...);
}

template <class... P, class... A>
inline cudaError_t launch_dependent(void (*f)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, A... args) {
  return launch_dependent_clusters(f, 1, grid, threads, smem, s, args...);
}

inline int targets_per_block(const PairConfig &c) { return c.tb / c.p * c.r; }

// `kernel` below is a SmoothingKernel (device.cuh).

// FP32 pair math, FP64 accumulation of per-tile partial sums.
bool pairs_f32_supported(const PairConfig &c, int kernel);
cudaError_t pairs_f32_occupancy(const PairConfig &c, bool diffusion, int kernel, int *blocks_per_sm);
// next_item: the work-item counter, zero at launch.  The packed tilings are the
// symmetric engine's (below): supported here, launched there.
cudaError_t launch_pairs_f32(const PairConfig &c, bool diffusion, int kernel, int grid,
                             const WorkItem *items, int n_items, const SegDesc *segs,
                             int *next_item, cudaStream_t s);

// The symmetric pair engine (FP32): each unordered pair once, sums into the
// items' slots; one block per item.  group: items over groups of kSymGroup
// tiles, else over single tile pairs.  sided: some items form one side's sums
// only (sharded systems).
cudaError_t sym_f32_occupancy(bool diffusion, int kernel, int *blocks_per_sm);
cudaError_t launch_sym_f32(bool group, bool sided, bool diffusion, int kernel, const SymItem *items, int n_items,
                           int sm_count, const SymSeg *segs, const int *jbase, double *slots, cudaStream_t s);
// Sums the slots of each listed tile into its rates.
cudaError_t launch_sym_sums(const SymSum *sums, int n_sums, const StageDesc *descs, const double *slots,
                            cudaStream_t s);

// FP64 with the same algebra as the FP32 kernel ("tuned FP64"), on the symmetric
// engine whatever the tiling.
bool pairs_f64_supported(const PairConfig &c, int kernel);
cudaError_t sym_f64_occupancy(bool diffusion, int kernel, int *blocks_per_sm);
cudaError_t launch_sym_f64(bool group, bool sided, bool diffusion, int kernel, const SymItem *items, int n_items,
                           int sm_count, const SymSeg *segs, const int *jbase, double *slots, cudaStream_t s);

// FP64, the reference's formula term by term (pow, divisions): the plain
// FP64 comparator.
bool pairs_plain_supported(const PairConfig &c, int kernel);
cudaError_t pairs_plain_occupancy(const PairConfig &c, int kernel, int *blocks_per_sm);
cudaError_t launch_pairs_plain(const PairConfig &c, int kernel, int grid, const WorkItem *items,
                               int n_items, const SegDesc *segs, int *next_item, cudaStream_t s);

// Per-particle stage kernel (RK4 stage update from the summed rates, pack).
cudaError_t launch_stage(int mode, int n_blocks, const StageItem *items, const StageDesc *descs,
                         cudaStream_t s);

// The same for a symmetric plan whose slots one wave wrote: sums each listed
// tile's slots and applies the stage (every mode but STAGE_PACK, STAGE_SHARD).
cudaError_t launch_sum_stage(int mode, int n_sums, const SymSum *sums, const StageDesc *descs,
                             const double *slots, cudaStream_t s);

// Diagnostics of one system.  `scratch` holds at least diag_scratch_doubles(n)
// doubles; out[0..10] = total vorticity (3), linear impulse (3), angular
// impulse (3), enstrophy, helicity; out[11] = kinetic energy.
size_t diag_scratch_doubles(int n);
cudaError_t launch_diagnostics(int n, int kernel, const double4 *pos64, const double4 *vor64,
                               const int *wake_id, double *scratch, double *out, bool quadratic,
                               cudaStream_t s);

// Vorticity field (FP64) of one system: field[3i..3i+2] = sum_j Z_ij alpha_j.
// part: influence_chunks(n) x 3n doubles of scratch (unused when that is 1).
int influence_chunks(int n);
cudaError_t launch_influence(int n, int kernel, const double4 *pos64, const double4 *vor64, double *part,
                             double *field, cudaStream_t s);
// Most columns per block of the columns kernel; a launch covers at most
// 65,535 x kInfluenceColumnGroup columns (the grid's y extent).
constexpr int kInfluenceColumnGroup = 32;
// The same for ncols strength vectors over one set of positions and radii:
// cols and field are ncols blocks of N x 3 doubles, part influence_chunks(n)
// times that; column c of field is bit-identical to launch_influence with
// vor64 = column c of cols.
cudaError_t launch_influence_columns(int n, int ncols, int kernel, const double4 *pos64, const double *cols,
                                     double *part, double *field, cudaStream_t s);

// Throughput probes: FP32 FFMA and FP64 DFMA chains.  flops = launched FMAs * 2.
cudaError_t launch_ffma_peak(int blocks, int threads, int iters, float *sink, cudaStream_t s);
cudaError_t launch_dfma_peak(int blocks, int threads, int iters, double *sink, cudaStream_t s);
// FMAs launched: as above (kPeakChains FMAs per thread and repetition, in pairs).
cudaError_t launch_ffma2_peak(int blocks, int threads, int iters, float *sink, cudaStream_t s);
constexpr int kPeakChains = 8;

}  // namespace pawan
