"""The symmetric pair engine (each unordered pair once) at the edges of its
decomposition: single tile pairs up to 256 tiles of 128 particles, groups of
four tiles beyond, the last tile and group full, one particle short and one
particle long."""
import numpy as np
import pytest

import oracle
from pawan_b200 import Batch, Server, System
from pawan_b200 import geometry as g
from pawan_b200.shard import ShardedSystem
from helpers import TOL_F32_MAX, TOL_F32_RMS, max_rel, rms_rel
from test_gpu_shard import emulated_rk4

pytestmark = pytest.mark.gpu

EDGE = 256 * 128  # the largest system in single tile pairs


def particles(n, mixed=False, seed=81):
    """A ring pair cut to n particles, its boxes at every distance class; with
    `mixed` alternating radii (no uniform-radius tile pair)."""
    sc = g.ring_pair(n_stations=-(-n // 16), seed=seed, nu=1e-3)
    pos, vor, rad, vol = (a[:n].copy() for a in sc.union())
    if mixed:
        rad[1::2] *= 0.8
    return pos, vor, rad, vol


def solved(ctx, arrays, nu, kernel="highorder"):
    s = System(ctx, [arrays[2].size], nu, "f32")
    s.set_kernel(kernel)
    s.set_particles(*arrays)
    s.solve()
    return s


@pytest.mark.parametrize("n", [64, 129, 1408, 1409, 2048])
@pytest.mark.parametrize("kernel", ["highorder", "gaussian"])
def test_launch_shapes_agree(ctx, n, kernel):
    """Tile pairs in a cluster of two blocks (alone, up to 74 of them), in one
    block of eight warps (up to 148) and in one of four (in a batch of more):
    bit for bit."""
    alone, systems = [], []
    for k in range(4):
        s = solved(ctx, particles(n, mixed=k % 2 == 1, seed=96 + k), 1e-3, kernel)
        alone.append(s.get_rates())
        systems.append(s)
    systems.append(solved(ctx, particles(3000, seed=95), 1e-3, kernel))  # 300 tile pairs
    alone.append(systems[-1].get_rates())
    Batch(ctx, systems).solve()
    for s, r in zip(systems, alone):
        assert np.array_equal(s.get_rates(), r)


@pytest.mark.parametrize("kernel", ["highorder", "gaussian"])
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", [383, 385, EDGE, EDGE + 1, EDGE + 511, EDGE + 512])
def test_against_restatement(ctx, n, mixed, kernel):
    """Sampled targets (the first, the last and 254 others) against the FP64
    restatement over all sources; repeated solves bit for bit."""
    arrays = particles(n, mixed)
    t = np.unique(np.concatenate([[0, n - 1], np.random.default_rng(n).choice(n, 254, replace=False)]))
    for nu in (1e-3, 0.0):
        s = solved(ctx, arrays, nu, kernel)
        u, da = s.union_rates()
        s.solve()
        u2, da2 = s.union_rates()
        assert np.array_equal(u, u2) and np.array_equal(da, da2)
        u_ref, da_ref = oracle.pairs(*arrays, nu, targets=t, kernel=kernel)
        assert rms_rel(u[t], u_ref) <= TOL_F32_RMS and max_rel(u[t], u_ref) <= TOL_F32_MAX
        assert rms_rel(da[t], da_ref) <= TOL_F32_RMS and max_rel(da[t], da_ref) <= TOL_F32_MAX
        s.close()


def test_batch_of_both_decompositions_matches_alone(ctx):
    """Systems on either side of the edge in one launch sequence: with a packed
    tiling set, all on the symmetric engine; untuned, those of more than 8,192
    particles on the one-sided kernel."""
    sizes = [EDGE + 1, 129, 2000, 8192, 8193]
    alone, systems = [], []
    for k, n in enumerate(sizes):
        arrays = particles(n, seed=90 + k)
        s = solved(ctx, arrays, 1e-3)
        alone.append(s.get_rates())
        systems.append(s)
    b = Batch(ctx, systems)
    b.solve()
    for n, s, r in zip(sizes, systems, alone):
        got = s.get_rates()
        assert np.array_equal(got, r) == (n <= 8192)
        assert rms_rel(got, r) <= TOL_F32_RMS
    b.set_config(128, unroll=4, packed=2)
    b.solve()
    for s, r in zip(systems, alone):
        assert np.array_equal(s.get_rates(), r)  # a system's slots and their order are its own


def test_untuned_batch_steps_both_kinds_of_system(ctx):
    """Per-system dt, graph and eager, over the two plans of an untuned batch."""
    scs = [g.single_ring(n_stations=k, seed=95 + k, nu=1e-3) for k in (1100, 40, 1030)]  # N = 8,800, 320, 8,240
    dts = np.array([0.001, 0.002, 0.003])
    runs = []
    for graph in (False, True):
        systems = [System.from_scenario(ctx, sc, "f32") for sc in scs]
        Batch(ctx, systems).rk4(dts, 2, use_graph=graph)
        runs.append([s.get_states() for s in systems])
    for sc, dt, a, b in zip(scs, dts, *runs):
        assert np.array_equal(a, b)
        solo = System.from_scenario(ctx, sc, "f32")
        solo.rk4(dt, 2)
        st0 = sc.state()
        assert rms_rel(a - st0, solo.get_states() - st0) <= TOL_F32_RMS


def test_sharded_groups_match_unsharded(ctx):
    """Emulated ranks of a system in groups: only the grouping of the FP64 sums
    may differ from the unsharded run."""
    sc = g.ring_pair(n_stations=2080, seed=83, nu=1e-3)  # N = 33,280: a ragged last block
    ref = System.from_scenario(ctx, sc, "f32")
    ref.rk4(sc.dt, 1)
    systems = [System.from_scenario(ctx, sc, "f32") for _ in range(2)]
    shards = [ShardedSystem(s, r, 2, gather=lambda recv, send: None) for r, s in enumerate(systems)]
    emulated_rk4(shards, sc.dt, 1)
    a, b = (s.get_states() for s in systems)
    assert np.array_equal(a, b)
    st0 = sc.state()
    assert rms_rel(a - st0, ref.get_states() - st0) < 1e-12


def test_served_slices_of_groups_match_alone(ctx):
    """A request in groups advancing by slices of its stages' items."""
    sc = g.ring_pair(n_stations=2100, seed=84, nu=1e-3, steps=2)  # N = 33,600
    srv = Server(ctx, budget_bytes=8 << 30, iteration_seconds=1e-4)
    rid = srv.submit_scenario(sc)[1]
    assert srv.wait(rid, 120)
    out = srv.fetch(rid)[0]
    assert srv.stats()["iterations"] > 8
    srv.close()
    solo = System.from_scenario(ctx, sc, "f32")
    solo.rk4(sc.dt, sc.steps)
    st0 = sc.state()
    assert rms_rel(out - st0, solo.get_states() - st0) < 1e-12
