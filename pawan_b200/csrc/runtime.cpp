// Host engine of the pawan B200 library: tile choices, execution plans over
// one or many systems (the reference's __interaction with its wakes), pair and
// stage launches, RK4 driving with CUDA graphs, autotuning internals, and a
// system's device buffers and state conversions.  The C ABI over it is in
// abi.cpp.
#include "runtime.h"

#include <nvtx3/nvToolsExt.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdint>
#include <cstring>
#include <numeric>

using namespace pawan;

namespace pawan {

int fail(pawan_ctx *ctx, int code, const std::string &msg) {
  if (ctx) ctx->err = msg;
  return code;
}

int cuda_fail(pawan_ctx *ctx, cudaError_t e, const char *where) {
  std::string m = std::string(where) + ": " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")";
  if (e == cudaErrorMemoryAllocation) return fail(ctx, PAWAN_ERR_NOMEM, m);
  return fail(ctx, PAWAN_ERR_CUDA, m);
}

TileChoice default_tile(int precision) {
  TileChoice t;
  if (precision == PAWAN_PREC_F32) {
    t.pc = PairConfig{128, 1, 4, 1, 0, 2};  // the symmetric engine
  } else {
    t.pc = PairConfig{128, 1, 1};
  }
  t.items_per_slot = 32;
  return t;
}

std::vector<TileChoice> tile_candidates(int precision, int kernel) {
  std::vector<TileChoice> v;
  if (precision == PAWAN_PREC_F32) {
    // (threads per target, targets per thread, unroll, blocks per SM, packed):
    // the scalar tilings as compiled in pair_f32.cu (0 = the default register
    // bound), the packed ones all the symmetric engine's
    const int shapes[][5] = {{1, 1, 4, 0, 0}, {2, 1, 4, 0, 0}, {4, 1, 4, 0, 0}, {1, 2, 1, 0, 0},
                             {1, 2, 2, 0, 0}, {1, 1, 4, 5, 0}, {1, 1, 1, 0, 1}, {1, 1, 2, 0, 1},
                             {1, 1, 4, 0, 1}, {1, 1, 2, 5, 1}, {1, 1, 2, 0, 2}, {1, 1, 4, 0, 2}};
    for (int tb : {128, 256})
      for (const auto &sh : shapes) {
        TileChoice t;
        t.pc = PairConfig{tb, sh[0], sh[2], sh[1], sh[3], sh[4]};
        if (pairs_f32_supported(t.pc, kernel)) v.push_back(t);
      }
    for (int split : {1, 2})
      for (int tb : {128, 256})
        for (int pk : {1, 2}) {
          TileChoice t;
          t.pc = PairConfig{tb, 1, 4, 1, 0, pk, split};
          if (pairs_f32_supported(t.pc, kernel)) v.push_back(t);
        }
  } else {
    for (int tb : {128, 256}) {
      TileChoice t;
      t.pc = PairConfig{tb, 1, 1};
      v.push_back(t);
    }
  }
  return v;
}

Plan::~Plan() { drop_graph(); }

void Plan::drop_graph() {
  if (graph_exec) cudaGraphExecDestroy(graph_exec);
  if (graph) cudaGraphDestroy(graph);
  graph_exec = nullptr;
  graph = nullptr;
}

bool Plan::stale() const {
  for (size_t s = 0; s < systems.size(); ++s)
    if (systems[s]->nu != nus[s] || systems[s]->geometry_version != geometry_versions[s])
      return true;
  return false;
}

bool tile_symmetric(int precision, const PairConfig &pc) {
  return precision == PAWAN_PREC_F64 || (precision == PAWAN_PREC_F32 && pc.packed > 0 && !pc.onesided);
}

static int occupancy(pawan_ctx *ctx, int precision, const PairConfig &pc, bool diffusion,
                     int kernel, int *bps) {
  cudaError_t e;
  if (precision == PAWAN_PREC_F32)
    e = pairs_f32_occupancy(pc, diffusion, kernel, bps);
  else
    e = pairs_plain_occupancy(pc, kernel, bps);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "occupancy query");
  if (*bps < 1) return fail(ctx, PAWAN_ERR_INVALID, "pair kernel does not fit on an SM");
  return PAWAN_OK;
}

bool tile_supported(int precision, const PairConfig &pc, int kernel) {
  if (precision == PAWAN_PREC_F32) return pairs_f32_supported(pc, kernel);
  if (precision == PAWAN_PREC_F64) return pairs_f64_supported(pc, kernel);
  return pairs_plain_supported(pc, kernel);
}

static_assert(PAWAN_KERNEL_HIGHORDER == KERNEL_HIGHORDER && PAWAN_KERNEL_GAUSSIAN == KERNEL_GAUSSIAN,
              "public and device smoothing-kernel codes agree");

static size_t shard_first(const pawan_system *y) { return (size_t)y->shard.rank * y->shard.size; }

static size_t shard_count(const pawan_system *y) {
  const size_t f = shard_first(y);
  return f >= y->n ? 0 : std::min(y->shard.size, y->n - f);
}

// ---- symmetric pair engine: work decomposition ----
// A system of up to kSymTilesMax tiles is covered by single tile pairs (enough
// blocks to fill the device from a few thousand particles on), a larger one by
// groups of kSymGroup tiles, whose sums are written once per four tile pairs.
constexpr int kSymTilesMax = 256;
// Bound on one system's slots: the rows of groups (or tiles) are processed in
// phases, the slots of a phase summed into the rates before the next reuses them.
// (One row's slots are the least: 6 KB per 128 particles, and as much again.)
constexpr double kSymSlotBytes = 2.0e9;
// Bound on the slots of all systems of a plan (or one phase of one of them): plans
// over more run in waves that reuse them.  512 ragged rings of 512 to 16,384
// particles hold 7.4e9 bytes in one wave.
constexpr double kPlanSlotBytes = 8.0e9;

namespace {

// The decomposition of one system: groups of g tiles, the runs of column groups
// per row, and the phases' row ranges [rows[p], rows[p + 1]).
struct SymLayout {
  int g = 1, ng = 0, run = 1;
  std::vector<int> rows;
  int runs(int a) const { return (ng - a + run - 1) / run; }
  // slots of group t in the phase of rows [r0, r1)
  int slots(int t, int r0, int r1) const {
    return std::max(0, std::min(t, r1) - r0) + (t >= r0 && t < r1 ? runs(t) : 0);
  }
};

SymLayout sym_layout(size_t n, int items_per_slot, double bytes, int world = 1) {
  SymLayout l;
  const int nt = (int)((n + kSymTile - 1) / kSymTile);
  l.g = nt <= kSymTilesMax ? 1 : kSymGroup;
  l.ng = (nt + l.g - 1) / l.g;
  if (l.g > 1) {
    // longer runs write fewer target-side sums; at least some dozens of items
    // per resident block (444 of them) keep the last ones from trailing (a rank of
    // a sharded system has its share of the pairs, most of them twice)
    const double pairs = 0.5 * (double)l.ng * (double)(l.ng + 1) * std::min(1.0, 2.0 / world);
    l.run = std::max(1, std::min(4, (int)(pairs / (444.0 * std::max(1, items_per_slot)))));
  }
  const double slot = 48.0 * kSymTile * l.g;
  l.rows.push_back(0);
  int r0 = 0;
  while (r0 < l.ng) {
    int r1 = r0;
    double used = 0.0;  // row a adds its runs and one slot per later group
    while (r1 < l.ng) {
      const double more = slot * (double)(l.runs(r1) + l.ng - 1 - r1);
      if (r1 > r0 && used + more > bytes) break;
      used += more;
      ++r1;
    }
    l.rows.push_back(r1);
    r0 = r1;
  }
  return l;
}

}  // namespace

double sym_slot_bytes(size_t n, double bytes) {
  const SymLayout l = sym_layout(n, 32, bytes);
  double most = 0.0;
  for (size_t p = 0; p + 1 < l.rows.size(); ++p) {
    double c = 0.0;
    for (int t = 0; t < l.ng; ++t) c += l.slots(t, l.rows[p], l.rows[p + 1]);
    most = std::max(most, c);
  }
  return most * 48.0 * kSymTile * l.g;
}

namespace {

// Whether this process computes particles of group t of a system (all of them
// when it is not sharded; block starts are multiples of a group).
bool sym_owned(const pawan_system *y, const SymLayout &l, int t) {
  if (!y->shard.active) return true;
  const size_t per = (size_t)kSymTile * l.g, f = shard_first(y);
  return t * per < f + shard_count(y) && (t + 1) * per > f;
}

// The systems' decompositions, and which phases of which systems share a wave:
// a wave's slots are summed before the next wave reuses them.
struct SymWaves {
  struct Unit {
    size_t system;
    int phase;
  };
  std::vector<SymLayout> lay;
  std::vector<std::vector<Unit>> waves;  // systems with the most tiles first
  double bytes = 0.0;                    // of the largest wave's slots
};

SymWaves sym_waves(const Plan &p, double system_bytes, double plan_bytes) {
  SymWaves w;
  for (auto *y : p.systems)
    w.lay.push_back(sym_layout(y->n, p.tile.items_per_slot, system_bytes, y->shard.active ? y->shard.world : 1));
  std::vector<size_t> order(p.systems.size());
  std::iota(order.begin(), order.end(), (size_t)0);
  std::stable_sort(order.begin(), order.end(),
                   [&](size_t a, size_t b) { return p.systems[a]->n > p.systems[b]->n; });
  std::vector<double> used;  // bytes of each wave
  for (size_t s : order) {
    const SymLayout &l = w.lay[s];
    size_t k = 0;  // a system's phases in waves of increasing number
    for (size_t ph = 0; ph + 1 < l.rows.size(); ++ph, ++k) {
      double need = 0.0;
      for (int t = 0; t < l.ng; ++t)
        if (sym_owned(p.systems[s], l, t)) need += l.slots(t, l.rows[ph], l.rows[ph + 1]);
      need *= 48.0 * kSymTile * l.g;
      while (k < used.size() && used[k] > 0.0 && used[k] + need > plan_bytes) ++k;
      if (k == used.size()) {
        used.push_back(0.0);
        w.waves.emplace_back();
      }
      used[k] += need;
      w.bytes = std::max(w.bytes, used[k]);
      w.waves[k].push_back({s, (int)ph});
    }
  }
  return w;
}

}  // namespace

// At least `count` doubles of slots.  The larger buffer is taken before the old one
// is given back, or, where both do not fit, after it.
static int reserve_slots(pawan_ctx *ctx, SlotPool &pool, size_t count) {
  if (pool.buf.n >= count) return PAWAN_OK;
  DBuf<double> larger;
  if (pool.buf.ordered) larger.ordered_on(pool.buf.stream);
  cudaError_t e = larger.alloc(count);
  if (e == cudaErrorMemoryAllocation && pool.buf.p) {
    const size_t had = pool.buf.n;
    pool.buf.reset();
    if (pool.buf.ordered) cudaStreamSynchronize(pool.buf.stream);
    e = larger.alloc(count);
    if (e != cudaSuccess) pool.buf.alloc(had);  // the other plans' (at worst at their next launch)
  }
  if (e != cudaSuccess) return cuda_fail(ctx, e, "pair-sum slots");
  std::swap(pool.buf.p, larger.p);
  std::swap(pool.buf.n, larger.n);
  return PAWAN_OK;
}

// Items, slots and sums of a plan on the symmetric engine.  A system's
// decomposition depends on its own size and the tiling only, so its arithmetic
// does not depend on the other systems of the plan.
static int build_sym_work(pawan_ctx *ctx, Plan &p, const SymWaves &w) {
  struct Costed {
    SymItem w;
    double cost;
  };
  std::vector<SymItem> items;
  std::vector<SymSum> sums;
  std::vector<int> jbase;
  const size_t n_waves = w.waves.size();
  p.waves.assign(n_waves, Plan::Wave{});
  for (size_t k = 0; k < n_waves; ++k) {
    Plan::Wave &P = p.waves[k];
    P.sum0 = (int)sums.size();
    size_t used[2] = {0, 0};  // slots so far: single-tile systems, grouped ones
    // items in launch order: those with tile pairs next to the diagonal, which take
    // longest, before a system's others
    std::vector<Costed> mine[2];
    std::vector<SymSum> of_tiles;
    for (const SymWaves::Unit &unit : w.waves[k]) {
      const size_t s = unit.system;
      const int ph = unit.phase;
      const SymLayout &l = w.lay[s];
      const pawan_system *y = p.systems[s];
      const int grouped = l.g > 1 ? 1 : 0, per = kSymTile * l.g;
      const int n = (int)y->n, nt = (n + kSymTile - 1) / kSymTile;
      const int r0 = l.rows[ph], r1 = l.rows[ph + 1];
      auto owned = [&](int t) { return sym_owned(y, l, t); };
      auto particles = [&](int t) { return (double)(std::min(n, (t + 1) * per) - t * per); };
      const int jb = (int)jbase.size();
      std::vector<int> i0(l.ng, -1);
      for (int t = 0; t < l.ng; ++t) {
        const int c = l.slots(t, r0, r1);
        if (!owned(t) || c == 0) {
          jbase.push_back(kNoSlot);
          continue;
        }
        const size_t first = used[grouped];
        used[grouped] += (size_t)c;
        if (used[grouped] > (size_t)INT32_MAX / 2) return fail(ctx, PAWAN_ERR_INVALID, "too many work items");
        jbase.push_back(t > r0 ? (int)first - r0 : kNoSlot);
        if (t >= r0 && t < r1) i0[t] = (int)first + (t - r0);
        for (int q = 0; q < l.g && t * l.g + q < nt; ++q) {
          const long long at = (long long)first * 6 * per + (long long)q * 6 * kSymTile;
          (grouped ? sums : of_tiles).push_back(SymSum{at, 6 * per, c, (int)s, t * l.g + q, ph > 0 ? 1 : 0});
        }
      }
      std::vector<Costed> late;
      for (int a = r0; a < r1; ++a) {
        int run = 0;
        for (int first = a; first < l.ng; first += l.run, ++run) {
          int b0 = first, b1 = std::min(l.ng, first + l.run);
          if (!owned(a)) {  // of the run the groups of this process alone (neighbours)
            while (b0 < b1 && !owned(b0)) ++b0;
            while (b0 < b1 && !owned(b1 - 1)) --b1;
            if (b0 == b1) continue;
          }
          double cost = 0.0;  // interactions credited: ordered pairs of owned targets
          bool sources = false;
          for (int b = b0; b < b1; ++b) {
            sources = sources || owned(b);
            const double both = particles(a) * particles(b);
            cost += (owned(a) ? both : 0.0) + (b != a && owned(b) ? both : 0.0);
          }
          const int side = !owned(a) ? SIDE_J : sources ? SIDE_BOTH : SIDE_I;
          if (side != SIDE_BOTH) p.sided = true;
          const Costed c{SymItem{(int)s, a, b0, b1, i0[a] < 0 ? kNoSlot : i0[a] + run, jb, side}, cost};
          if (b0 <= a + (l.g > 1 ? 1 : 2))
            mine[grouped].push_back(c);
          else
            late.push_back(c);
        }
      }
      mine[grouped].insert(mine[grouped].end(), late.begin(), late.end());
    }
    P.groups = (int)mine[1].size();
    P.tiles = (int)mine[0].size();
    for (int grouped : {1, 0})
      for (const Costed &c : mine[grouped]) {
        items.push_back(c.w);
        p.item_costs.push_back(c.cost);
      }
    // the single-tile items' slots lie behind the groups'
    P.tile_slots = used[1] * 6 * kSymTile * kSymGroup;
    for (SymSum &t : of_tiles) t.first += (long long)P.tile_slots;
    sums.insert(sums.end(), of_tiles.begin(), of_tiles.end());
    P.sums = (int)sums.size() - P.sum0;
    p.slot_count = std::max(p.slot_count, P.tile_slots + used[0] * 6 * kSymTile);
  }
  for (const SymSum &s : sums) p.slot_bytes += (double)s.count * 48.0 * kSymTile;
  if (items.size() > (size_t)INT32_MAX) return fail(ctx, PAWAN_ERR_INVALID, "too many work items");
  p.n_items = (int)items.size();
  std::vector<SymSeg> segs;
  for (size_t s = 0; s < p.systems.size(); ++s) {
    const pawan_system *y = p.systems[s];
    const StageDesc &g = p.stage_host[s];
    segs.push_back(SymSeg{g.pos32, g.vor32, g.poslo, g.vorlo, g.pos64, g.vor64, g.boxes,
                          (int)y->n, y->nu, (float)(y->r_near * y->r_near)});
  }
  PAWAN_TRY(reserve_slots(ctx, *p.pool, p.slot_count));
  PAWAN_CUDA(ctx, p.sym_items.alloc(items.size()));
  PAWAN_CUDA(ctx, p.sym_segs.alloc(segs.size()));
  PAWAN_CUDA(ctx, p.sym_jbase.alloc(jbase.size()));
  PAWAN_CUDA(ctx, p.sym_sums.alloc(sums.size()));
  PAWAN_CUDA(ctx, cudaMemcpyAsync(p.sym_items.p, items.data(), items.size() * sizeof(SymItem),
                                  cudaMemcpyHostToDevice, ctx->stream));
  PAWAN_CUDA(ctx, cudaMemcpyAsync(p.sym_segs.p, segs.data(), segs.size() * sizeof(SymSeg),
                                  cudaMemcpyHostToDevice, ctx->stream));
  PAWAN_CUDA(ctx, cudaMemcpyAsync(p.sym_jbase.p, jbase.data(), jbase.size() * sizeof(int),
                                  cudaMemcpyHostToDevice, ctx->stream));
  PAWAN_CUDA(ctx, cudaMemcpyAsync(p.sym_sums.p, sums.data(), sums.size() * sizeof(SymSum),
                                  cudaMemcpyHostToDevice, ctx->stream));
  return PAWAN_OK;
}

// Work decomposition.  Target tiles of tb/p particles; sources in chunks of
// whole tb-tiles sized so that the launch holds about `items_per_slot` items
// per resident block (or of `fixed_chunk_sources` when > 0, which makes a
// system's arithmetic independent of the other systems in the plan).  The
// systems with the largest items come first, so the dynamic counter hands out
// the long items early (longest-processing-time order), and within a system a
// target tile's chunks are consecutive.
int build_plan(pawan_ctx *ctx, const std::vector<pawan_system *> &systems, int precision,
               const TileChoice &tile, std::unique_ptr<Plan> &out, int fixed_chunk_sources,
               const PlanMemory &memory) {
  if (systems.empty()) return fail(ctx, PAWAN_ERR_INVALID, "plan over no systems");
  const int kernel = systems[0]->kernel;
  for (auto *s : systems)
    if (s->kernel != kernel)
      return fail(ctx, PAWAN_ERR_INVALID, "systems of one plan must share the smoothing kernel");
  if (!tile_supported(precision, tile.pc, kernel))
    return fail(ctx, PAWAN_ERR_INVALID, "unsupported pair tiling for this precision and kernel");
  std::unique_ptr<Plan> p(new Plan());
  p->systems = systems;
  p->precision = precision;
  p->kernel = kernel;
  p->tile = tile;
  for (auto *s : systems) {
    p->nus.push_back(s->nu);
    p->geometry_versions.push_back(s->geometry_version);
    p->box_versions.push_back(~0ull);
    if (s->nu != 0.0) p->diffusion = true;
    const double targets = s->shard.active ? (double)shard_count(s) : (double)s->n;
    p->interactions += targets * (double)s->n;
  }
  int bps = 0;
  SymWaves waves;
  p->sym = tile_symmetric(precision, tile.pc);
  if (p->sym) {
    cudaError_t e = precision == PAWAN_PREC_F64 ? sym_f64_occupancy(p->diffusion, kernel, &bps)
                                                : sym_f32_occupancy(p->diffusion, kernel, &bps);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "occupancy query");
    if (bps < 1) return fail(ctx, PAWAN_ERR_INVALID, "pair kernel does not fit on an SM");
    if (!memory.own_slots) p->pool = ctx->slots.lock();
    if (!p->pool) {
      p->pool = std::make_shared<SlotPool>();
      if (memory.ordered) p->pool->buf.ordered_on(ctx->stream);
      if (!memory.own_slots) ctx->slots = p->pool;
    }
    // Where the device has no room for the slots, in more and smaller phases and
    // waves, down to one row of tiles at a time.
    double share = 1.0, before = -1.0;
    for (;;) {
      waves = sym_waves(*p, share * (memory.system_bytes > 0.0 ? memory.system_bytes : kSymSlotBytes),
                        share * (memory.plan_bytes > 0.0 ? memory.plan_bytes : kPlanSlotBytes));
      const int st = waves.bytes == before ? PAWAN_ERR_NOMEM
                                           : reserve_slots(ctx, *p->pool, (size_t)(waves.bytes / sizeof(double)));
      if (st == PAWAN_OK) break;
      if (st != PAWAN_ERR_NOMEM || share < 1e-4) return st;
      before = waves.bytes;
      share *= 0.25;
    }
    p->fused_sums = waves.waves.size() == 1;
    for (auto *s : systems)
      if (s->shard.active) p->fused_sums = false;
  } else {
    PAWAN_TRY(occupancy(ctx, precision, tile.pc, p->diffusion, kernel, &bps));
  }
  p->grid = ctx->sm_count * bps;
  const int TB = p->sym ? kSymTile : tile.pc.tb;
  const int TPB = p->sym ? kSymTile : targets_per_block(tile.pc);
  const double slots = (double)p->grid;
  const double target_pairs =
      std::max(p->interactions / (slots * std::max(1, tile.items_per_slot)), (double)TPB * TB);

  struct ItemCost {
    WorkItem w;
    double cost;
  };
  std::vector<ItemCost> items;
  // per system: partial slots [target tiles][chunks][6][TPB] (none with one
  // chunk), rates [6][n] (none where the stage sums the slots), one counter per
  // target tile (one-sided kernels)
  if (TPB % 8 != 0) return fail(ctx, PAWAN_ERR_INVALID, "targets per block must be a multiple of 8");
  size_t partial_total = 0, box_total = 0, rates_total = 0, count_total = 0;
  std::vector<size_t> partial_off(systems.size()), box_off(systems.size());
  std::vector<size_t> rates_off(systems.size()), count_off(systems.size());
  std::vector<double> sys_cost(systems.size(), 0.0);
  p->nchunks.resize(systems.size());
  for (size_t s = 0; s < systems.size(); ++s) {
    const int n = (int)systems[s]->n;
    const int src_tiles = (n + TB - 1) / TB;
    int tiles_per_chunk = fixed_chunk_sources > 0
                              ? (fixed_chunk_sources + TB - 1) / TB
                              : (int)std::ceil(target_pairs / ((double)TPB * TB));
    tiles_per_chunk = std::max(1, std::min(tiles_per_chunk, src_tiles));
    const int nch = p->sym ? 1 : (src_tiles + tiles_per_chunk - 1) / tiles_per_chunk;
    p->nchunks[s] = nch;
    const size_t target_tiles = ((size_t)n + TPB - 1) / TPB;
    partial_off[s] = partial_total;
    if (nch > 1) partial_total += target_tiles * (size_t)nch * 6 * (size_t)TPB;
    rates_off[s] = rates_total;
    if (!p->fused_sums) rates_total += 6 * (size_t)n;
    count_off[s] = count_total;
    if (!p->sym) count_total += target_tiles;
    box_off[s] = box_total;
    box_total += 2 * (size_t)src_tiles;
    // targets: all particles, or this process's block of a sharded system
    // (block starts are multiples of kShardAlign, so of every TPB and TB)
    const pawan_system *y = systems[s];
    const int t_lo = y->shard.active ? (int)shard_first(y) : 0;
    const int t_hi = y->shard.active ? t_lo + (int)shard_count(y) : n;
    // target-major: a target tile's chunks are consecutive, so they run at
    // about the same time and the block completing the tile finds their
    // partial slots still in L2
    for (int t0 = t_lo; t0 < t_hi && !p->sym; t0 += TPB) {
      const int nt = std::min(TPB, t_hi - t0);
      for (int c = 0; c < nch; ++c) {
        const int s0 = c * tiles_per_chunk * TB;
        const int s1 = std::min(n, (c + 1) * tiles_per_chunk * TB);
        const double cost = (double)nt * (double)(s1 - s0);
        sys_cost[s] = std::max(sys_cost[s], cost);
        items.push_back({WorkItem{(int)s, t0, c, s0, s1}, cost});
      }
    }
  }
  // Systems whose items are largest go first (longest-processing-time order
  // across the systems of a batch); each system's items keep their order.
  std::stable_sort(items.begin(), items.end(), [&](const ItemCost &a, const ItemCost &b) {
    return sys_cost[a.w.seg] > sys_cost[b.w.seg];
  });
  if (items.size() > (size_t)INT32_MAX) return fail(ctx, PAWAN_ERR_INVALID, "too many work items");
  p->n_items = (int)items.size();

  if (memory.ordered) {
    p->partial.ordered_on(ctx->stream);
    p->rates.ordered_on(ctx->stream);
    p->tile_count.ordered_on(ctx->stream);
    p->boxes.ordered_on(ctx->stream);
    p->items.ordered_on(ctx->stream);
    p->segs.ordered_on(ctx->stream);
    p->stage_items.ordered_on(ctx->stream);
    p->shard_items.ordered_on(ctx->stream);
    p->stage_descs.ordered_on(ctx->stream);
    p->sym_items.ordered_on(ctx->stream);
    p->sym_segs.ordered_on(ctx->stream);
    p->sym_jbase.ordered_on(ctx->stream);
    p->sym_sums.ordered_on(ctx->stream);
  }
  PAWAN_CUDA(ctx, p->partial.alloc(partial_total));
  // the pair kernels discard the slots' L2 lines after summing them: every
  // slot must start on a 128-byte line (slot sizes are multiples of 128 bytes)
  if (reinterpret_cast<uintptr_t>(p->partial.p) % 128 != 0)
    return fail(ctx, PAWAN_ERR_CUDA, "partial-sum buffer not 128-byte aligned");
  PAWAN_CUDA(ctx, p->rates.alloc(rates_total));
  PAWAN_CUDA(ctx, p->tile_count.alloc(count_total));
  if (count_total > 0)
    PAWAN_CUDA(ctx, cudaMemsetAsync(p->tile_count.p, 0, p->tile_count.bytes(), ctx->stream));
  PAWAN_CUDA(ctx, p->boxes.alloc(box_total));
  std::vector<WorkItem> wh(items.size());
  p->item_costs.resize(items.size());
  for (size_t k = 0; k < items.size(); ++k) {
    wh[k] = items[k].w;
    p->item_costs[k] = items[k].cost;  // target x source pairs of the item
  }
  std::vector<SegDesc> sh(systems.size());
  std::vector<StageItem> sih, shh;
  p->stage_host.resize(systems.size());
  for (size_t s = 0; s < systems.size(); ++s) {
    pawan_system *y = systems[s];
    SegDesc &d = sh[s];
    d.pos32 = y->pos32.p;
    d.vor32 = y->vor32.p;
    d.poslo = y->poslo.p;
    d.vorlo = y->vorlo.p;
    d.pos64 = y->pos64.p;
    d.vor64 = y->vor64.p;
    d.boxes = p->boxes.p + box_off[s];
    d.partial = p->nchunks[s] > 1 ? p->partial.p + partial_off[s] : nullptr;
    d.rates = rates_total > 0 ? p->rates.p + rates_off[s] : nullptr;
    d.tile_count = count_total > 0 ? p->tile_count.p + count_off[s] : nullptr;
    d.n = (int)y->n;
    d.nchunks = p->nchunks[s];
    d.nu = y->nu;
    d.near2 = (float)(y->r_near * y->r_near);
    StageDesc &g = p->stage_host[s];
    g.rates = d.rates;
    g.n = d.n;
    g.X = y->X.p;
    g.Xs = y->Xs.p;
    g.K1 = y->K1.p;
    g.K2 = y->K2.p;
    g.R = y->R.p;
    g.rad = y->rad.p;
    g.vol = y->vol.p;
    g.pos32 = y->pos32.p;
    g.vor32 = y->vor32.p;
    g.poslo = y->poslo.p;
    g.vorlo = y->vorlo.p;
    g.pos64 = y->pos64.p;
    g.vor64 = y->vor64.p;
    g.boxes = p->boxes.p + box_off[s];
    g.box_tile = TB;
    g.ox = y->ox;
    g.oy = y->oy;
    g.oz = y->oz;
    g.dt = 0.0;
    g.xchg_out = y->shard.active ? y->shard.send : nullptr;
    g.xchg_in = y->shard.active ? y->shard.recv : nullptr;
    g.shard = y->shard.active ? (int)y->shard.size : 0;
    g.shard_first = y->shard.active ? (int)shard_first(y) : 0;
    for (int l0 = 0; l0 < d.n; l0 += kStageThreads) sih.push_back(StageItem{(int)s, l0});
    if (y->shard.active) {
      const int f = (int)shard_first(y), e = f + (int)shard_count(y);
      for (int l0 = f; l0 < e; l0 += kStageThreads) shh.push_back(StageItem{(int)s, l0});
    }
  }
  p->n_stage_blocks = (int)sih.size();
  p->n_shard_blocks = (int)shh.size();
  p->dts.assign(systems.size(), 0.0);
  if (p->sym) PAWAN_TRY(build_sym_work(ctx, *p, waves));
  PAWAN_CUDA(ctx, p->items.alloc(wh.size()));
  PAWAN_CUDA(ctx, p->segs.alloc(sh.size()));
  PAWAN_CUDA(ctx, p->stage_items.alloc(sih.size()));
  PAWAN_CUDA(ctx, p->stage_descs.alloc(sh.size()));
  if (!wh.empty())
    PAWAN_CUDA(ctx, cudaMemcpyAsync(p->items.p, wh.data(), wh.size() * sizeof(WorkItem),
                                    cudaMemcpyHostToDevice, ctx->stream));
  PAWAN_CUDA(ctx, cudaMemcpyAsync(p->segs.p, sh.data(), sh.size() * sizeof(SegDesc),
                                  cudaMemcpyHostToDevice, ctx->stream));
  PAWAN_CUDA(ctx, cudaMemcpyAsync(p->stage_items.p, sih.data(), sih.size() * sizeof(StageItem),
                                  cudaMemcpyHostToDevice, ctx->stream));
  if (!shh.empty()) {
    PAWAN_CUDA(ctx, p->shard_items.alloc(shh.size()));
    PAWAN_CUDA(ctx, cudaMemcpyAsync(p->shard_items.p, shh.data(), shh.size() * sizeof(StageItem),
                                    cudaMemcpyHostToDevice, ctx->stream));
  }
  PAWAN_CUDA(ctx, cudaMemcpyAsync(p->stage_descs.p, p->stage_host.data(),
                                  p->stage_host.size() * sizeof(StageDesc), cudaMemcpyHostToDevice,
                                  ctx->stream));
  out = std::move(p);
  // the plan's tile boxes: repack the current states (idempotent for the
  // packed arrays, which already hold pack(X) between API calls)
  PAWAN_TRY(launch_stage_mode(ctx, *out, STAGE_PACK));
  // (the host tables were staged by the copies above; an ordered plan is used
  // on the same stream, so only the others wait here)
  if (!memory.ordered) PAWAN_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return PAWAN_OK;
}

int check_dts(pawan_ctx *ctx, size_t n, const double *dt, double dt0) {
  for (size_t s = 0; s < n; ++s) {
    const double v = dt ? dt[s] : dt0;
    if (!(v > 0.0) || !std::isfinite(v)) return fail(ctx, PAWAN_ERR_INVALID, "dt must be positive");
  }
  return PAWAN_OK;
}

// Puts each system's dt into the device stage table (only when it changed).  A
// rejected call changes nothing: what p.dts holds is always what the table holds.
int set_plan_dt(pawan_ctx *ctx, Plan &p, const double *dt, double dt0) {
  PAWAN_TRY(check_dts(ctx, p.systems.size(), dt, dt0));
  bool changed = false;
  for (size_t s = 0; s < p.systems.size(); ++s) {
    const double v = dt ? dt[s] : dt0;
    p.stage_host[s].dt = v;
    changed = changed || p.dts[s] != v;
  }
  if (changed) {
    PAWAN_CUDA(ctx, cudaMemcpyAsync(p.stage_descs.p, p.stage_host.data(),
                                    p.stage_host.size() * sizeof(StageDesc),
                                    cudaMemcpyHostToDevice, ctx->stream));
    for (size_t s = 0; s < p.systems.size(); ++s) p.dts[s] = p.stage_host[s].dt;
  }
  return PAWAN_OK;
}

static cudaEvent_t take_event(pawan_ctx *ctx) {
  if (!ctx->event_pool.empty()) {
    cudaEvent_t e = ctx->event_pool.back();
    ctx->event_pool.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  if (cudaEventCreate(&e) != cudaSuccess) return nullptr;
  return e;
}

// Work items [first, first + count) of a plan on the symmetric engine, and the
// slot sums of every wave whose last item is among them.
static int launch_sym_range(pawan_ctx *ctx, Plan &p, int first, int count) {
  PAWAN_TRY(reserve_slots(ctx, *p.pool, p.slot_count));
  int at = 0;
  for (const Plan::Wave &ph : p.waves) {
    for (bool group : {true, false}) {
      const int n = group ? ph.groups : ph.tiles;
      const int lo = std::max(first, at), hi = std::min(first + count, at + n);
      at += n;
      if (lo >= hi) continue;
      double *slots = p.pool->buf.p + (group ? 0 : ph.tile_slots);
      const auto launch = p.precision == PAWAN_PREC_F64 ? launch_sym_f64 : launch_sym_f32;
      PAWAN_CUDA(ctx, launch(group, p.sided, p.diffusion, p.kernel, p.sym_items.p + lo, hi - lo, ctx->sm_count,
                             p.sym_segs.p, p.sym_jbase.p, slots, ctx->stream));
      ctx->launches++;
    }
    if (!p.fused_sums && at > first && at <= first + count) {
      PAWAN_CUDA(ctx, launch_sym_sums(p.sym_sums.p + ph.sum0, ph.sums, p.stage_descs.p, p.pool->buf.p, ctx->stream));
      ctx->launches++;
    }
  }
  return PAWAN_OK;
}

int launch_pairs(pawan_ctx *ctx, Plan &p, bool allow_events) {
  return launch_pairs_range(ctx, p, 0, p.n_items, allow_events);
}

int launch_pairs_range(pawan_ctx *ctx, Plan &p, int first, int count, bool allow_events) {
  if (first < 0 || count < 0 || first + count > p.n_items)
    return fail(ctx, PAWAN_ERR_INVALID, "work-item range outside the plan");
  const WorkItem *items = p.items.p + first;
  for (size_t s = 0; s < p.systems.size(); ++s)
    if (p.box_versions[s] != p.systems[s]->pack_version) {
      // another plan repacked these systems since this plan's boxes were made
      PAWAN_TRY(launch_stage_mode(ctx, p, STAGE_PACK));
      break;
    }
  if (!p.sym) PAWAN_CUDA(ctx, cudaMemsetAsync(ctx->d_counter, 0, sizeof(int), ctx->stream));
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (ctx->profile && allow_events) {
    e0 = take_event(ctx);
    e1 = take_event(ctx);
    if (!e0 || !e1) return fail(ctx, PAWAN_ERR_CUDA, "cannot create profiling events");
    PAWAN_CUDA(ctx, cudaEventRecord(e0, ctx->stream));
  }
  cudaError_t e = cudaSuccess;
  if (p.sym)
    PAWAN_TRY(launch_sym_range(ctx, p, first, count));
  else if (p.precision == PAWAN_PREC_F32)
    e = launch_pairs_f32(p.tile.pc, p.diffusion, p.kernel, p.grid, items, count, p.segs.p,
                         ctx->d_counter, ctx->stream);
  else
    e = launch_pairs_plain(p.tile.pc, p.kernel, p.grid, items, count, p.segs.p, ctx->d_counter,
                           ctx->stream);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "pair kernel launch");
  if (!p.sym) ctx->launches++;
  if (e0) {
    PAWAN_CUDA(ctx, cudaEventRecord(e1, ctx->stream));
    ctx->pending.push_back({e0, e1});
    ctx->pair_launches++;
    double work = 0.0;
    for (int i = first; i < first + count; ++i) work += p.item_costs[i];
    ctx->pair_interactions += work;
  }
  return PAWAN_OK;
}

static void note_repack(Plan &p) {
  for (size_t s = 0; s < p.systems.size(); ++s) {
    p.systems[s]->pack_version++;
    p.box_versions[s] = p.systems[s]->pack_version;
  }
}

// Algorithmic HBM bytes of one stage launch: per particle the rates (48 bytes:
// the pair kernel's summed chunks, or the gathered rates of a sharded system; all
// slots of 48 bytes where the stage sums them itself), the FP64 state vectors the
// mode reads and writes, radius and volume, and the 128 bytes of packed FP32 /
// FP64 tile data; 32 bytes of bounding box per tile.  An RK4 stage is 288-336
// bytes per particle beside the rates or slots.
static double stage_bytes(const Plan &p, int mode) {
  double total = 0.0;
  for (size_t s = 0; s < p.systems.size(); ++s) {
    const pawan_system *y = p.systems[s];
    const double n = (double)y->n;
    const double rates = 48.0;
    const double pack = 16.0 + 128.0 + 32.0 / (double)p.stage_host[s].box_tile;
    double per = 0.0;
    switch (mode) {
      case STAGE_RATES: per = rates + 48.0; break;
      case STAGE_K1: case STAGE_K2: per = rates + 48.0 + 96.0 + pack; break;
      case STAGE_K3: per = rates + 96.0 + 96.0 + pack; break;
      case STAGE_FINAL: per = rates + 144.0 + 48.0 + pack; break;
      case STAGE_EULER: per = rates + 48.0 + 48.0 + pack; break;
      case STAGE_PACK: per = 48.0 + pack; break;
      default: per = 0.0;
    }
    total += n * per;
  }
  if (p.fused_sums && mode != STAGE_PACK) {
    for (const pawan_system *y : p.systems) total -= 48.0 * (double)y->n;
    total += p.slot_bytes;
  }
  return total;
}

int launch_stage_mode(pawan_ctx *ctx, Plan &p, int mode) {
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (ctx->profile) {
    e0 = take_event(ctx);
    e1 = take_event(ctx);
    if (!e0 || !e1) return fail(ctx, PAWAN_ERR_CUDA, "cannot create profiling events");
    PAWAN_CUDA(ctx, cudaEventRecord(e0, ctx->stream));
  }
  cudaError_t e = p.fused_sums && mode != STAGE_PACK
                      ? launch_sum_stage(mode, p.waves[0].sums, p.sym_sums.p, p.stage_descs.p, p.pool->buf.p, ctx->stream)
                      : launch_stage(mode, p.n_stage_blocks, p.stage_items.p, p.stage_descs.p, ctx->stream);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "stage kernel launch");
  ctx->launches++;
  if (e0) {
    PAWAN_CUDA(ctx, cudaEventRecord(e1, ctx->stream));
    ctx->stage_pending.push_back({e0, e1});
    ctx->stage_launches++;
    ctx->stage_bytes += stage_bytes(p, mode);
  }
  if (mode != STAGE_RATES) note_repack(p);
  return PAWAN_OK;
}

// NVTX range over a scope (header-only NVTX; a no-op unless a profiler is
// attached): one per RK4 step and one per stage, so a timeline shows the
// reference's stage structure (rk4.cpp:24-66).
struct NvtxRange {
  explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
};

static int rk4_one_step(pawan_ctx *ctx, Plan &p, bool allow_events) {
  static const int modes[4] = {STAGE_K1, STAGE_K2, STAGE_K3, STAGE_FINAL};
  static const char *names[4] = {"pawan rk4 k1", "pawan rk4 k2", "pawan rk4 k3", "pawan rk4 k4+update"};
  NvtxRange step("pawan rk4 step");
  for (int s = 0; s < 4; ++s) {
    NvtxRange stage(names[s]);
    PAWAN_TRY(launch_pairs(ctx, p, allow_events));
    PAWAN_TRY(launch_stage_mode(ctx, p, modes[s]));
  }
  return PAWAN_OK;
}

int rk4_steps(pawan_ctx *ctx, Plan &p, size_t nsteps, bool use_graph) {
  if (!use_graph) {
    for (size_t k = 0; k < nsteps; ++k) PAWAN_TRY(rk4_one_step(ctx, p, true));
    return PAWAN_OK;
  }
  if (p.sym) {
    // (a captured graph holds the slots' address: nothing can be reserved under
    // capture, and a plan that needed more has moved them)
    PAWAN_TRY(reserve_slots(ctx, *p.pool, p.slot_count));
    if (p.graph_exec && p.graph_slots != p.pool->buf.p) p.drop_graph();
    p.graph_slots = p.pool->buf.p;
  }
  if (!p.graph_exec) {
    for (size_t s = 0; s < p.systems.size(); ++s)
      if (p.box_versions[s] != p.systems[s]->pack_version) {
        PAWAN_TRY(launch_stage_mode(ctx, p, STAGE_PACK));
        break;
      }
    PAWAN_CUDA(ctx, cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    const unsigned long long before = ctx->launches.load();
    int st = rk4_one_step(ctx, p, false);
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(ctx->stream, &g);
    p.graph_kernels = ctx->launches.load() - before;
    ctx->launches = before;  // capture enqueues nothing; replays count below
    if (st != PAWAN_OK) {
      if (g) cudaGraphDestroy(g);
      return st;
    }
    if (e != cudaSuccess) return cuda_fail(ctx, e, "graph capture");
    p.graph = g;
    PAWAN_CUDA(ctx, cudaGraphInstantiate(&p.graph_exec, g, 0));
  }
  for (size_t k = 0; k < nsteps; ++k) {
    for (size_t s = 0; s < p.systems.size(); ++s)
      if (p.box_versions[s] != p.systems[s]->pack_version) {
        PAWAN_TRY(launch_stage_mode(ctx, p, STAGE_PACK));
        break;
      }
    PAWAN_CUDA(ctx, cudaGraphLaunch(p.graph_exec, ctx->stream));
    ctx->launches += p.graph_kernels;
    for (int st = 0; st < 4; ++st) note_repack(p);
  }
  return PAWAN_OK;
}

int autotune_plan(pawan_ctx *ctx, const std::vector<pawan_system *> &systems, int precision,
                  TileChoice *best) {
  cudaEvent_t e0, e1;
  PAWAN_CUDA(ctx, cudaEventCreate(&e0));
  PAWAN_CUDA(ctx, cudaEventCreate(&e1));
  double best_ms = 1e300;
  TileChoice best_t = default_tile(precision);
  int status = PAWAN_OK;
  // One right-hand side as an RK4 stage runs it: the pair launch and the
  // reduction of its chunk partials (STAGE_RATES writes only the rates
  // buffer), so that finer chunking pays for the partials it adds.
  auto rhs = [&](Plan &p) -> int {
    PAWAN_TRY(launch_pairs(ctx, p, false));
    return launch_stage_mode(ctx, p, STAGE_RATES);
  };
  auto time_tile = [&](const TileChoice &t, double *ms) -> int {
    std::unique_ptr<Plan> p;
    PAWAN_TRY(build_plan(ctx, systems, precision, t, p));
    PAWAN_TRY(rhs(*p));  // warm-up
    PAWAN_CUDA(ctx, cudaEventRecord(e0, ctx->stream));
    const int reps = 2;
    for (int r = 0; r < reps; ++r) PAWAN_TRY(rhs(*p));
    PAWAN_CUDA(ctx, cudaEventRecord(e1, ctx->stream));
    PAWAN_CUDA(ctx, cudaEventSynchronize(e1));
    float f = 0.f;
    PAWAN_CUDA(ctx, cudaEventElapsedTime(&f, e0, e1));
    *ms = f / reps;
    return PAWAN_OK;
  };
  // A tiling whose buffers do not fit beside what the device holds is no candidate.
  bool any = false;
  auto candidate = [&](const TileChoice &t) -> int {
    double ms = 0;
    const int st = time_tile(t, &ms);
    if (st != PAWAN_OK) return st;
    any = true;
    if (ms < best_ms) {
      best_ms = ms;
      best_t = t;
    }
    return PAWAN_OK;
  };
  // 1) tile shape at the default chunking, 2) chunking for the best shape.
  bool sym_timed = false;
  for (TileChoice t : tile_candidates(precision, systems[0]->kernel)) {
    if (tile_symmetric(precision, t.pc)) {
      // one engine behind all of them: timed once, as the default tiling
      if (sym_timed) continue;
      sym_timed = true;
      t.pc = default_tile(precision).pc;
    }
    status = candidate(t);
    if (status != PAWAN_OK && status != PAWAN_ERR_NOMEM) break;
  }
  if (any && (status == PAWAN_OK || status == PAWAN_ERR_NOMEM)) {
    const TileChoice shape = best_t;
    for (int ips : kTuneItemsPerSlot) {
      TileChoice t = shape;
      t.items_per_slot = ips;
      status = candidate(t);
      if (status != PAWAN_OK && status != PAWAN_ERR_NOMEM) break;
    }
    if (status == PAWAN_ERR_NOMEM) status = PAWAN_OK;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (status == PAWAN_OK) *best = best_t;
  return status;
}

int system_alloc(pawan_system *sys) {
  pawan_ctx *ctx = sys->ctx;
  const size_t n = sys->n;
  if (sys->ordered_alloc) {
    for (auto *b : {&sys->X, &sys->Xs, &sys->K1, &sys->K2, &sys->R, &sys->rad, &sys->vol,
                    &sys->diag_scratch, &sys->diag_out, &sys->Xc, &sys->field, &sys->columns})
      b->ordered_on(ctx->stream);
    sys->wake_id.ordered_on(ctx->stream);
    for (auto *b : {&sys->pos32, &sys->vor32, &sys->poslo, &sys->vorlo}) b->ordered_on(ctx->stream);
    sys->pos64.ordered_on(ctx->stream);
    sys->vor64.ordered_on(ctx->stream);
  }
  PAWAN_CUDA(ctx, sys->X.alloc(6 * n));
  PAWAN_CUDA(ctx, sys->Xs.alloc(6 * n));
  PAWAN_CUDA(ctx, sys->K1.alloc(6 * n));
  PAWAN_CUDA(ctx, sys->K2.alloc(6 * n));
  PAWAN_CUDA(ctx, sys->R.alloc(6 * n));
  PAWAN_CUDA(ctx, sys->rad.alloc(n));
  PAWAN_CUDA(ctx, sys->vol.alloc(n));
  PAWAN_CUDA(ctx, sys->wake_id.alloc(n));
  PAWAN_CUDA(ctx, sys->pos32.alloc(n));
  PAWAN_CUDA(ctx, sys->vor32.alloc(n));
  PAWAN_CUDA(ctx, sys->poslo.alloc(n));
  PAWAN_CUDA(ctx, sys->vorlo.alloc(n));
  PAWAN_CUDA(ctx, sys->pos64.alloc(n));
  PAWAN_CUDA(ctx, sys->vor64.alloc(n));
  PAWAN_CUDA(ctx, sys->diag_scratch.alloc(diag_scratch_doubles((int)n)));
  PAWAN_CUDA(ctx, sys->diag_out.alloc(12));
  std::vector<int> wid(n);
  for (size_t w = 0; w < sys->counts.size(); ++w)
    for (size_t i = 0; i < sys->counts[w]; ++i) wid[sys->offsets[w] + i] = (int)w;
  // on the context's (non-blocking) stream, so later copies on it are ordered after these
  PAWAN_CUDA(ctx, cudaMemcpyAsync(sys->wake_id.p, wid.data(), n * sizeof(int),
                                  cudaMemcpyHostToDevice, ctx->stream));
  PAWAN_CUDA(ctx, cudaMemsetAsync(sys->X.p, 0, 6 * n * sizeof(double), ctx->stream));
  // (the pageable wake ids were staged by the copy; ordered systems are only
  // used on this stream)
  if (!sys->ordered_alloc) PAWAN_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return PAWAN_OK;
}

int system_ensure_plan(pawan_system *sys) {
  if (!sys->has_particles)
    return fail(sys->ctx, PAWAN_ERR_STATE, "particles not set (pawan_system_set_particles)");
  if (sys->plan && !sys->plan->stale() && sys->plan->tile == sys->tile &&
      sys->plan->precision == sys->precision)
    return PAWAN_OK;
  sys->plan.reset();
  return build_plan(sys->ctx, {sys}, sys->precision, sys->tile, sys->plan);
}

static std::vector<HostCopy> state_copies(const pawan_system *sys, double *dev, double *host) {
  std::vector<HostCopy> v;
  for (size_t w = 0; w < sys->counts.size(); ++w) {
    const size_t o = sys->offsets[w], c = sys->counts[w];
    v.push_back({dev + 3 * o, host + 6 * o, 3 * c * sizeof(double)});
    v.push_back({dev + 3 * sys->n + 3 * o, host + 6 * o + 3 * c, 3 * c * sizeof(double)});
  }
  return v;
}

// Reference layout (per wake [x | alpha]) -> device union layout [x | alpha].
int state_to_device(pawan_system *sys, const double *state) {
  return copy_to_device(sys->ctx, state_copies(sys, sys->X.p, const_cast<double *>(state)));
}

// Device union layout -> reference layout; synchronous.
int state_from_device(pawan_system *sys, const double *dev_union, double *state) {
  return copy_to_host(sys->ctx, state_copies(sys, const_cast<double *>(dev_union), state));
}

}  // namespace pawan
