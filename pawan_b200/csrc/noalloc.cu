// pawan_interact_noalloc: the FP32 all-pairs interaction for callers that
// cannot allocate device memory.
//
// Who needs it: code that runs where cudaMalloc is not allowed or not safe --
// inside a host callback, under a memory manager that owns every allocation on
// the device (a pool handed to a plugin), or in a hard real-time loop where an
// allocation's implicit synchronisation and latency are unacceptable.  Such a
// caller owns its inputs and outputs but cannot let the library create
// buffers.  This entry point therefore keeps all of its working memory (the
// packed FP32 tile data, tile bounding boxes, per-chunk partial sums, the
// work list, the per-tile counters, the summed rates and the scheduler
// counter) in one file-scope device array,
// `g_noalloc_scratch`, sized for at most kNoallocMaxParticles particles.
// Every GPU that loads the library reserves that array until the process
// exits.
//
// Set-up: the first call on a device (with that device current) looks up the
// array's device address with cudaGetSymbolAddress and caches it; make that
// first call before any stream capture.  Later calls only launch kernels.
// All calls share the one array, so calls whose kernels overlap on the GPU
// (different streams, different host threads) race and must be serialised by
// the caller.  Whatever must start at zero (the scheduler counter and the
// per-tile counters) is cleared by the call itself, the count of finished
// prepare blocks by the last of them (the array starts zeroed) and once more by
// the call's last kernel, so that calls that raced leave nothing wrong for the
// calls after them; the rest is fully overwritten before it is read.
//
// The pair kernel is the one-sided FP32 kernel (pair_f32.cu) with the high-order
// smoothing kernel only, where pawan_system_solve runs the symmetric engine by
// default: the array holds 512 slots of 128 targets, and that engine takes t^2 of
// them for t tiles, so they would do up to 22 tiles (2,816 particles).  A system of
// t tiles is split into 512 / t source chunks, and several threads share a target's
// sources (noalloc_config below): a few thousand particles fill the device that
// way.  With one thread per target and fixed chunks of 4,096 sources, one call at
// N = 4,096 ran 32 blocks for 540 us, now 75, 58 of them in the pair kernel
// (N = 16,384: 560 us, now 513).  The FP32 positions are taken
// relative to particle 0 (pawan_system_set_particles uses the centroid), and
// the near-tile radius max(4 s_max, 0.03 x extent) measures the extent from
// particle 0, so it can be up to twice the allocating path's: more tile pairs
// may take the accurate near formulation.  Results therefore agree with
// pawan_system_solve within the FP32 tolerance, not bit for bit.
#include <cmath>
#include <cstddef>
#include <mutex>

#include "../../include/pawan_b200.h"
#include "device.cuh"
#include "kernels.h"

namespace pawan {
namespace {

constexpr int kNoallocMaxParticles = 16384;
constexpr int kNaTB = 128;         // threads per block = sources per tile
constexpr int kNaMaxTiles = (kNoallocMaxParticles + kNaTB - 1) / kNaTB;
constexpr int kNaSlots = 512;      // chunk slots of kNaTB targets
constexpr int kNaMaxP = 4;         // most threads per target
constexpr int kNaMaxItems = kNaSlots * kNaMaxP;
constexpr int kNaPrepBlocks = (kNoallocMaxParticles + kStageThreads - 1) / kStageThreads;

// Layout of the scratch array.  The kernels need 16-byte alignment of the
// float4 arrays (their offsets are multiples of 256 bytes) and natural
// alignment of the rest.
struct NoallocScratch {
  float4 pos32[kNoallocMaxParticles];
  float4 vor32[kNoallocMaxParticles];
  float4 poslo[kNoallocMaxParticles];
  float4 vorlo[kNoallocMaxParticles];
  float4 boxes[2 * kNaMaxTiles];
  double partial[kNaSlots * 6 * kNaTB];                    // [target tile][chunk][6][targets]
  double rates[6 * kNoallocMaxParticles];                  // [6][n]
  float block_max[2 * kNaPrepBlocks];  // per prepare block: max s, max |x - x0|^2
  WorkItem items[kNaMaxItems];
  int tile_count[kNaMaxTiles * kNaMaxP];
  SegDesc seg;
  int counter;
  int prepared;  // blocks of the current call's prepare launch done; 0 between calls
};

// The tiling and the source chunk of a call.  Threads per target: 4 up to 4,096
// particles, 2 beyond (pair kernel at N = 2,048: 27 us with 4, 30 with 2, 47
// with 1; at 4,096: 58, 60 and 68; at 8,192: 156, 145 and 155).
struct NoallocConfig {
  PairConfig pc;
  int chunk;   // sources per work item: whole tiles
  int chunks;
  int tiles;   // target tiles
};

NoallocConfig noalloc_config(int n) {
  NoallocConfig c;
  const int st = (n + kNaTB - 1) / kNaTB;
  c.pc = PairConfig{kNaTB, n <= 4096 ? 4 : 2, 4};
  const int most = kNaSlots / st;               // chunks that the slots hold
  const int per = (st + most - 1) / most;       // source tiles per chunk
  c.chunk = per * kNaTB;
  c.chunks = (st + per - 1) / per;
  c.tiles = (n + targets_per_block(c.pc) - 1) / targets_per_block(c.pc);
  return c;
}

static_assert(sizeof(NoallocScratch) < 5050000, "the array is 5.0 MB, as pawan_b200.h says");
static_assert(offsetof(NoallocScratch, boxes) % 256 == 0 && offsetof(NoallocScratch, partial) % 256 == 0 &&
                  offsetof(NoallocScratch, rates) % 256 == 0,
              "scratch arrays on 256-byte boundaries");

static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(NoallocScratch)];

// Pack: positions relative to particle 0 as FP32 hi/lo, strengths hi/lo,
// s^2/2 and volume; the bounding box (with the range of s^2/2 in w) of each
// 128-particle tile; per-block maxima of the smoothing radius and of the
// distance from particle 0.  The last block to finish then writes the
// near-tile radius (the rule of pawan_system_set_particles, with the extent
// measured from particle 0), the segment descriptor and the work list, and
// clears the counters.
__global__ void __launch_bounds__(kStageThreads)
    noalloc_prepare(NoallocScratch *S, const double *pos, const double *vor, const double *rad,
                    const double *vol, int n, double nu, int tpb, int tiles, int chunk, int chunks) {
  __shared__ int s_last;
  __shared__ float lo[4][kStageThreads], hi[4][kStageThreads];
  __shared__ float ms[kStageThreads], me[kStageThreads];
  const int t = threadIdx.x;
  const int l = blockIdx.x * kStageThreads + t;
  const bool has = l < n;
  float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
  float s_l = 0.f, e2 = 0.f;
  if (has) {
    const double rx = pos[3 * l] - pos[0], ry = pos[3 * l + 1] - pos[1], rz = pos[3 * l + 2] - pos[2];
    const float hx = (float)rx, hy = (float)ry, hz = (float)rz;
    const double s = rad[l];
    const float ax = (float)vor[3 * l], ay = (float)vor[3 * l + 1], az = (float)vor[3 * l + 2];
    const float hw = (float)(0.5 * s * s);
    S->pos32[l] = make_float4(hx, hy, hz, hw);
    S->poslo[l] = make_float4((float)(rx - (double)hx), (float)(ry - (double)hy),
                              (float)(rz - (double)hz), 0.f);
    S->vor32[l] = make_float4(ax, ay, az, (float)vol[l]);
    S->vorlo[l] = make_float4((float)(vor[3 * l] - (double)ax), (float)(vor[3 * l + 1] - (double)ay),
                              (float)(vor[3 * l + 2] - (double)az), 0.f);
    p = make_float4(hx, hy, hz, hw);
    s_l = (float)s;
    e2 = (float)(rx * rx + ry * ry + rz * rz);
  }
  lo[0][t] = has ? p.x : INFINITY;
  lo[1][t] = has ? p.y : INFINITY;
  lo[2][t] = has ? p.z : INFINITY;
  lo[3][t] = has ? p.w : INFINITY;
  hi[0][t] = has ? p.x : -INFINITY;
  hi[1][t] = has ? p.y : -INFINITY;
  hi[2][t] = has ? p.z : -INFINITY;
  hi[3][t] = has ? p.w : -INFINITY;
  ms[t] = s_l;
  me[t] = e2;
  __syncthreads();
  for (int s = kStageThreads / 2; s > 0; s >>= 1) {
    if (t < s) {
      ms[t] = fmaxf(ms[t], ms[t + s]);
      me[t] = fmaxf(me[t], me[t + s]);
    }
    if ((t % kNaTB) < s && s < kNaTB) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        lo[k][t] = fminf(lo[k][t], lo[k][t + s]);
        hi[k][t] = fmaxf(hi[k][t], hi[k][t + s]);
      }
    }
    __syncthreads();
  }
  if ((t % kNaTB) == 0 && l < n) {
    const int b = l / kNaTB;
    S->boxes[2 * b] = make_float4(lo[0][t], lo[1][t], lo[2][t], lo[3][t]);
    S->boxes[2 * b + 1] = make_float4(hi[0][t], hi[1][t], hi[2][t], hi[3][t]);
  }
  if (t == 0) {
    S->block_max[2 * blockIdx.x] = ms[0];
    S->block_max[2 * blockIdx.x + 1] = me[0];
    __threadfence();
    s_last = atomicAdd(&S->prepared, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;  // block-uniform
  __threadfence();
  if (t == 0) {
    float a = 0.f, b = 0.f;
    for (int k = 0; k < (int)gridDim.x; ++k) {
      a = fmaxf(a, __ldcg(&S->block_max[2 * k]));
      b = fmaxf(b, __ldcg(&S->block_max[2 * k + 1]));
    }
    const float r_near = fmaxf(4.f * a, 0.03f * sqrtf(b));
    SegDesc d;
    d.pos32 = S->pos32;
    d.vor32 = S->vor32;
    d.poslo = S->poslo;
    d.vorlo = S->vorlo;
    d.pos64 = nullptr;
    d.vor64 = nullptr;
    d.boxes = S->boxes;
    d.partial = S->partial;
    d.rates = S->rates;
    d.tile_count = S->tile_count;
    d.n = n;
    d.nchunks = chunks;
    d.nu = nu;
    d.near2 = r_near * r_near;
    S->seg = d;
    S->counter = 0;
    S->prepared = 0;
  }
  for (int q = t; q < tiles; q += kStageThreads) S->tile_count[q] = 0;
  for (int it = t; it < tiles * chunks; it += kStageThreads) {
    const int q = it / chunks, c = it - q * chunks;
    S->items[it] = WorkItem{0, q * tpb, c, c * chunk, min(n, (c + 1) * chunk)};
  }
}

// The pair kernel's rates ([6][n], chunks summed in chunk order) into the
// caller's N x 3 outputs.  Clears the count of prepare blocks for the next call.
__global__ void noalloc_reduce(NoallocScratch *S, int n, double *vel, double *dvor) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l == 0) S->prepared = 0;
  if (l >= n) return;
  for (int k = 0; k < 3; ++k) {
    vel[3 * (size_t)l + k] = S->rates[(size_t)k * n + l];
    dvor[3 * (size_t)l + k] = S->rates[(size_t)(3 + k) * n + l];
  }
}

struct DeviceSlot {
  NoallocScratch *scratch = nullptr;
  int grid[2] = {0, 0};  // resident blocks with 2 and with 4 threads per target
};
constexpr int kMaxDevices = 64;
DeviceSlot g_slots[kMaxDevices];
std::mutex g_slots_mu;

// Once per device, with that device current: the array's device address (in
// host code the symbol itself names a host-side stand-in, not device memory)
// and the persistent grid size.
cudaError_t device_slot(int dev, DeviceSlot *out) {
  std::lock_guard<std::mutex> lk(g_slots_mu);
  DeviceSlot &s = g_slots[dev];
  if (!s.scratch) {
    void *ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    int sms = 0, bps = 0;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    for (int k = 0; k < 2; ++k) {
      int bps0 = 0;
      const PairConfig pc{kNaTB, k ? 4 : 2, 4};
      e = pairs_f32_occupancy(pc, true, KERNEL_HIGHORDER, &bps);
      if (e != cudaSuccess) return e;
      e = pairs_f32_occupancy(pc, false, KERNEL_HIGHORDER, &bps0);
      if (e != cudaSuccess) return e;
      s.grid[k] = sms * (bps < bps0 ? bps : bps0);
    }
    s.scratch = static_cast<NoallocScratch *>(ptr);
  }
  *out = s;
  return cudaSuccess;
}

}  // namespace
}  // namespace pawan

extern "C" int pawan_interact_noalloc(const double *position, const double *vorticity,
                                      const double *radius, const double *volume, size_t n,
                                      double nu, double *velocity, double *retvorcity,
                                      void *stream) {
  using namespace pawan;
  if (!position || !vorticity || !radius || !volume || !velocity || !retvorcity)
    return PAWAN_ERR_INVALID;
  if (n < 2 || n > (size_t)kNoallocMaxParticles || !std::isfinite(nu) || nu < 0.0)
    return PAWAN_ERR_INVALID;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return PAWAN_ERR_CUDA;
  DeviceSlot slot;
  if (device_slot(dev, &slot) != cudaSuccess) return PAWAN_ERR_CUDA;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int ni = (int)n;
  const int pblocks = (ni + kStageThreads - 1) / kStageThreads;
  const NoallocConfig c = noalloc_config(ni);
  noalloc_prepare<<<pblocks, kStageThreads, 0, s>>>(slot.scratch, position, vorticity, radius, volume, ni, nu,
                                                     targets_per_block(c.pc), c.tiles, c.chunk, c.chunks);
  const int items = c.tiles * c.chunks;
  const int resident = slot.grid[c.pc.p == 4 ? 1 : 0];
  cudaError_t e = launch_pairs_f32(c.pc, nu != 0.0, KERNEL_HIGHORDER, items < resident ? items : resident,
                                   slot.scratch->items, items, &slot.scratch->seg, &slot.scratch->counter, s);
  if (e != cudaSuccess) return PAWAN_ERR_CUDA;
  noalloc_reduce<<<(ni + 255) / 256, 256, 0, s>>>(slot.scratch, ni, velocity, retvorcity);
  if (cudaGetLastError() != cudaSuccess) return PAWAN_ERR_CUDA;
  return PAWAN_OK;
}
