// Smoothed vorticity field of a system, FP64: the counterpart of
// __interaction::influence (src/interaction/interaction.cpp:110-155), which
// __interaction::resolve (:45-47) runs for the influence-matrix path of
// __resolve::rebuild (src/resolve/resolve.cpp:10-57).
//
// Reference: every unordered pair once, INFLUENCE
// (src/interaction/interaction_utils.h:519-556) with
// sigma = sqrt((s_i^2 + s_j^2)/2), Z = ZETASIG(rho, sigma)
// (src/interaction/highorder.h:20-23), K_target += Z alpha_source and
// K_source += Z alpha_target; plus SELFINFLUENCE (:593-605),
// K_i += ZETASIG(0, s_i) alpha_i.  In gather form
//   K_i = sum_j Z(rho_ij, sigma_ij) alpha_j   over every j, i included:
// the j = i term has rho = 0 and sigma = s_i, which is SELFINFLUENCE.
// With w = (rho^2 + sigma^2)^(-1/2) and u = sigma^2 w^2 = 1/(rho_bar^2 + 1):
//   Z = (15 / 8 pi) sigma^-3 (rho_bar^2 + 1)^-7.5 = (15 / 8 pi) u^6 w^3,
// or with the Gaussian kernel (src/interaction/gaussian.h:20-23)
//   Z = exp(-rho_bar^2 / 2) / (sigma^3 (2 pi)^1.5).
//
// FP64 throughout keeps the resolve's linear solve as accurate as the
// reference's.
//
// Sources are cut into chunks by the system's size alone (chunk_sources: enough
// blocks for a full device from a thousand particles on, one chunk from 32,768
// on); a chunk is summed with FMAs in source order and the chunks in chunk
// order.  Both kernels follow that order and form Z with the same function,
// so a column of the batched kernel is bit-identical to a single field.
//
// The single-field kernel keeps one target per thread: 21 FP64 operations for
// Z and 3 FMAs per pair.  The columns kernel evaluates the field of many
// strength vectors over the same positions and radii at once -- the
// influence-matrix columns of __resolve::rebuild (resolve.cpp:19-31), which
// differ only in alpha -- as a matrix product: a block forms Z of 64 targets and
// 16 sources once, in shared memory, and each thread multiplies it into a
// register tile of 4 targets x 6 values (two columns' vectors), so a pair costs
// 3 FMAs per column and 21 / 32 of an operation for Z when a block covers all of
// 32 columns, and five 16-byte shared-memory loads feed 24 FMAs.  25 columns of
// 3,950 particles: 243 us on one B200 against 1,130 for one target per thread and
// eight columns per block (124 blocks).
#include <algorithm>

#include "device.cuh"
#include "kernels.h"
#include "rsqrt64.cuh"

namespace pawan {
namespace {

constexpr int kInfThreads = 128;
// columns kernel: register tile per thread, targets and sources per block step
constexpr int kTM = 4, kTN = 6, kRows = 16, kBT = kTM * kRows, kKT = 16;
constexpr int kValues = 3 * kInfluenceColumnGroup;  // most values (3 per column) of a block
static_assert(kValues % kTN == 0 && kTN % 3 == 0, "column groups are whole register tiles");

// Z(rho_ij, sigma_ij) for target i (position ri, hi = s_i^2 / 2) and source
// j (rj = position, smoothing radius); operations written out so that every
// kernel rounds them the same way.
template <int KERN>
__device__ __forceinline__ double pair_z(const double4 ri, double hi, const double4 rj) {
  const double dx = __dsub_rn(ri.x, rj.x), dy = __dsub_rn(ri.y, rj.y), dz = __dsub_rn(ri.z, rj.z);
  const double rho2 = __fma_rn(dz, dz, __fma_rn(dy, dy, __dmul_rn(dx, dx)));
  const double sig2 = __fma_rn(0.5 * rj.w, rj.w, hi);
  if (KERN == KERNEL_GAUSSIAN) {
    const double cg = 0.06349363593424096978;  // (2 pi)^-1.5
    const double is = rsqrt_f64_full(sig2);
    const double is2 = __dmul_rn(is, is);
    return __dmul_rn(__dmul_rn(exp(-0.5 * __dmul_rn(rho2, is2)), __dmul_rn(is2, is)), cg);
  } else {
    const double c = 1.875 * kInvPi;  // 15 / (8 pi)
    const double w = rsqrt_f64_full(__dadd_rn(rho2, sig2));
    const double w2 = __dmul_rn(w, w);
    const double u = __dmul_rn(sig2, w2);
    const double u2 = __dmul_rn(u, u);
    const double u6 = __dmul_rn(__dmul_rn(u2, u2), u2);
    return __dmul_rn(__dmul_rn(c, u6), __dmul_rn(w2, w));
  }
}

// Block (target block, chunk): sources [c * chunk, (c + 1) * chunk) into
// out[c][i][3].
template <int KERN>
__global__ void __launch_bounds__(kInfThreads)
    influence_kernel(int n, int chunk, const double4 *__restrict__ pos, const double4 *__restrict__ vor,
                     double *__restrict__ out) {
  __shared__ double4 sp[kInfThreads];
  __shared__ double4 sv[kInfThreads];
  const int tid = threadIdx.x;
  const int i = blockIdx.x * kInfThreads + tid;
  const int s0 = blockIdx.y * chunk, s1 = min(n, s0 + chunk);
  const bool valid = i < n;
  const double4 ri = valid ? pos[i] : make_double4(0.0, 0.0, 0.0, 1.0);
  const double hi = __dmul_rn(0.5 * ri.w, ri.w);
  double kx = 0.0, ky = 0.0, kz = 0.0;
  for (int ts = s0; ts < s1; ts += kInfThreads) {
    __syncthreads();
    const int j = ts + tid;
    if (j < s1) {
      sp[tid] = pos[j];
      sv[tid] = vor[j];
    }
    __syncthreads();
    const int cnt = min(kInfThreads, s1 - ts);
#pragma unroll 4
    for (int jj = 0; jj < cnt; ++jj) {
      const double4 aj = sv[jj];
      const double z = pair_z<KERN>(ri, hi, sp[jj]);
      kx = __fma_rn(z, aj.x, kx);
      ky = __fma_rn(z, aj.y, ky);
      kz = __fma_rn(z, aj.z, kz);
    }
  }
  if (valid) {
    double *o = out + 3 * ((size_t)blockIdx.y * n + i);
    o[0] = kx;
    o[1] = ky;
    o[2] = kz;
  }
}

__device__ __forceinline__ double4 tp_of(const double4 *pos, int n, int i) {
  return i < n ? pos[i] : make_double4(0.0, 0.0, 0.0, 1.0);
}

__device__ __forceinline__ void cp_async8(double *smem, const double *gmem) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(a), "l"(gmem) : "memory");
}

// Shared memory of a block: two stages of sources, strengths and Z.
struct ColumnStage {
  double4 sp[kKT];           // sources
  double sz[kKT][kBT];       // Z
  double sa[kKT * kValues];  // strengths: [source][value]
};

// Block (target block, value group, chunk).  cols is ncols blocks of N x 3
// doubles (column c, particle j, component k at (c*N + j)*3 + k), value v =
// 3 c + k; out has that layout per chunk.  blockDim = kRows x (values / kTN)
// threads for the product, rounded up to a multiple of kBT.
// While a step's product runs, the next step's sources and strengths arrive by
// asynchronous copies; its Z follows the product.
template <int KERN>
__global__ void __launch_bounds__(kRows * kValues / kTN, 2)
    influence_columns_kernel(int n, int ncols, int values, int chunk, const double4 *__restrict__ pos,
                             const double *__restrict__ cols, double *__restrict__ out) {
  __shared__ ColumnStage stage[2];
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int tc = values / kTN;  // threads across the values
  const int row = min(tid / tc, kRows - 1), col = tid - tid / tc * tc;
  const bool product = tid < kRows * tc;
  const int i0 = blockIdx.x * kBT;
  const int v0 = blockIdx.y * values;
  const int nv = min(values, 3 * ncols - v0);  // a whole number of columns
  const int s0 = blockIdx.z * chunk, s1 = min(n, s0 + chunk);
  const double *const mine = cols + (size_t)(v0 / 3) * n * 3;

  // sources [ts, ts + cnt) and their strengths: a column's are contiguous
  auto fetch = [&](ColumnStage &st, int ts) {
    const int e = 3 * min(kKT, s1 - ts);
    for (int q = tid; q < nv * kKT; q += nthr) {
      const int c = q / (3 * kKT), x = q - c * (3 * kKT), j = x / 3;
      if (x < e) cp_async8(&st.sa[j * values + 3 * c + (x - 3 * j)], mine + ((size_t)c * n + ts) * 3 + x);
    }
    for (int q = tid; q < 4 * min(kKT, s1 - ts); q += nthr)
      cp_async8(reinterpret_cast<double *>(st.sp) + q, reinterpret_cast<const double *>(pos + ts) + q);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // each thread keeps one target, and four sources' chains at a time
  const double4 ri = tp_of(pos, n, i0 + (tid & (kBT - 1)));
  const double hi = __dmul_rn(0.5 * ri.w, ri.w);
  auto form_z = [&](ColumnStage &st, int cnt) {
    const int i = tid & (kBT - 1), step = nthr / kBT;
    for (int j = tid / kBT; j < cnt; j += 4 * step) {
      double z[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) z[q] = pair_z<KERN>(ri, hi, st.sp[min(j + q * step, cnt - 1)]);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (j + q * step < cnt) st.sz[j + q * step][i] = z[q];
    }
  };
  auto wait = [] {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  };

  double acc[kTM][kTN];
#pragma unroll
  for (int a = 0; a < kTM; ++a)
#pragma unroll
    for (int b = 0; b < kTN; ++b) acc[a][b] = 0.0;
  fetch(stage[0], s0);
  wait();
  form_z(stage[0], min(kKT, s1 - s0));
  int cur = 0;
  for (int ts = s0; ts < s1; ts += kKT, cur ^= 1) {
    const ColumnStage &st = stage[cur];
    const int cnt = product ? min(kKT, s1 - ts) : 0;
    __syncthreads();  // this step's Z is whole; the other stage is no longer read
    if (ts + kKT < s1) fetch(stage[cur ^ 1], ts + kKT);
#pragma unroll 4
    for (int j = 0; j < cnt; ++j) {
      const double2 *zp = reinterpret_cast<const double2 *>(&st.sz[j][row * kTM]);
      const double2 *ap = reinterpret_cast<const double2 *>(&st.sa[j * values + col * kTN]);
      double z[kTM], a[kTN];
#pragma unroll
      for (int q = 0; q < kTM / 2; ++q) {
        const double2 v = zp[q];
        z[2 * q] = v.x;
        z[2 * q + 1] = v.y;
      }
#pragma unroll
      for (int q = 0; q < kTN / 2; ++q) {
        const double2 v = ap[q];
        a[2 * q] = v.x;
        a[2 * q + 1] = v.y;
      }
#pragma unroll
      for (int x = 0; x < kTM; ++x)
#pragma unroll
        for (int y = 0; y < kTN; ++y) acc[x][y] = __fma_rn(z[x], a[y], acc[x][y]);
    }
    if (ts + kKT < s1) {
      wait();
      form_z(stage[cur ^ 1], min(kKT, s1 - ts - kKT));
    }
  }
  if (!product) return;
  double *const base = out + (size_t)blockIdx.z * ncols * n * 3;
#pragma unroll
  for (int x = 0; x < kTM; ++x) {
    const int i = i0 + row * kTM + x;
    if (i >= n) continue;
#pragma unroll
    for (int y = 0; y < kTN; ++y) {
      const int v = col * kTN + y;  // within the group
      if (v >= nv) continue;
      const int c = (v0 + v) / 3, k = (v0 + v) - 3 * c;
      base[((size_t)c * n + i) * 3 + k] = acc[x][y];
    }
  }
}

// field[x] = part[0][x] + part[1][x] + ..., in that order.
__global__ void influence_sum_kernel(size_t count, int chunks, const double *__restrict__ part,
                                     double *__restrict__ field) {
  const size_t x = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= count) return;
  double r = part[x];
  for (int c = 1; c < chunks; ++c) r = __dadd_rn(r, part[(size_t)c * count + x]);
  field[x] = r;
}

// Sources per chunk, a function of n alone: about 32,768 / n chunks of at least
// 32 sources (128 targets per block: 256 blocks), one from 32,768 particles on.
int chunk_sources(int n) {
  const int want = std::max(1, (32768 + n - 1) / n);
  const int per = (n + want - 1) / want;
  return std::max(32, (per + 31) / 32 * 32);
}

cudaError_t sum_chunks(size_t count, int chunks, const double *part, double *field, cudaStream_t s) {
  influence_sum_kernel<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(count, chunks, part, field);
  return cudaGetLastError();
}

}  // namespace

int influence_chunks(int n) {
  const int per = chunk_sources(n);
  return (n + per - 1) / per;
}

cudaError_t launch_influence_columns(int n, int ncols, int kernel, const double4 *pos64, const double *cols,
                                     double *part, double *field, cudaStream_t s) {
  if (n <= 0 || ncols <= 0) return cudaSuccess;
  const int chunks = influence_chunks(n);
  const int total = 3 * ncols, groups = (total + kValues - 1) / kValues;
  if (groups > 65535) return cudaErrorInvalidValue;
  // equal groups, a whole number of register tiles each
  const int values = ((total + groups - 1) / groups + kTN - 1) / kTN * kTN;
  const dim3 grid((n + kBT - 1) / kBT, (total + values - 1) / values, chunks);
  const int threads = (kRows * (values / kTN) + kBT - 1) / kBT * kBT;
  double *out = chunks > 1 ? part : field;
  if (kernel == KERNEL_GAUSSIAN)
    influence_columns_kernel<KERNEL_GAUSSIAN>
        <<<grid, threads, 0, s>>>(n, ncols, values, chunk_sources(n), pos64, cols, out);
  else
    influence_columns_kernel<KERNEL_HIGHORDER>
        <<<grid, threads, 0, s>>>(n, ncols, values, chunk_sources(n), pos64, cols, out);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || chunks == 1) return e;
  return sum_chunks((size_t)ncols * n * 3, chunks, part, field, s);
}

cudaError_t launch_influence(int n, int kernel, const double4 *pos64, const double4 *vor64, double *part,
                             double *field, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int chunks = influence_chunks(n);
  const dim3 grid((n + kInfThreads - 1) / kInfThreads, chunks);
  double *out = chunks > 1 ? part : field;
  if (kernel == KERNEL_GAUSSIAN)
    influence_kernel<KERNEL_GAUSSIAN><<<grid, kInfThreads, 0, s>>>(n, chunk_sources(n), pos64, vor64, out);
  else
    influence_kernel<KERNEL_HIGHORDER><<<grid, kInfThreads, 0, s>>>(n, chunk_sources(n), pos64, vor64, out);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || chunks == 1) return e;
  return sum_chunks((size_t)n * 3, chunks, part, field, s);
}

}  // namespace pawan
