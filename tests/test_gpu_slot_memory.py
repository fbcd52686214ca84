"""Device memory of the symmetric engine's slots: bounded for a plan over many
systems, which then runs in waves, and shared by the plans of a context."""
import numpy as np
import pytest
import torch

from pawan_b200 import Batch, Context, Server, System
from pawan_b200 import geometry as g
from helpers import TOL_F32_RMS, rms_rel

pytestmark = pytest.mark.gpu


@pytest.fixture
def own():
    c = Context(0)
    yield c
    c.close()


def used_bytes():
    free, total = torch.cuda.mem_get_info()
    return total - free


def particles(n, seed):
    sc = g.ring_pair(n_stations=-(-n // 16), seed=seed, nu=1e-3)
    return [np.ascontiguousarray(a[:n]) for a in sc.union()]


# 24 x 32,768 particles in single tiles, 10 x 131,072 in groups of tiles: 9.7 and
# 10 GB of slots if they were all held at once
@pytest.mark.parametrize("n,count,prec", [(32768, 24, "f64"), (131072, 10, "f32")])
def test_a_batch_over_the_bound_runs_in_waves(own, n, count, prec):
    sizes = [n] * count + [2000, 129]
    arrays = [particles(k, 5) for k in (n, 2000, 129)]
    alone = []
    for a in arrays:
        s = System(own, [len(a[0])], 1e-3, prec)
        s.set_particles(*a)
        s.solve()
        alone.append(s.get_rates())
        s.close()
    systems = []
    for k in sizes:
        s = System(own, [k], 1e-3, prec)
        s.set_particles(*arrays[[n, 2000, 129].index(k)])
        systems.append(s)
    before = used_bytes()
    b = Batch(own, systems)
    if prec == "f32":
        b.set_config(128, unroll=4, packed=2, items_per_slot=32)  # the default, as the systems alone
    b.solve()
    # the slots' bound, and per particle the 48-byte rates, 24 of work tables and boxes
    assert used_bytes() - before <= 8.0e9 + 100.0 * sum(sizes) + (64 << 20)
    for k, s in zip(sizes, systems):
        assert np.array_equal(s.get_rates(), alone[[n, 2000, 129].index(k)])
    b.close()
    for s in systems:
        s.close()


def test_systems_of_a_context_share_their_slots(own):
    a = particles(32768, 6)
    systems = []
    before = 0
    for k in range(8):
        s = System(own, [32768], 1e-3, "f32")
        s.set_particles(*a)
        s.solve()
        systems.append(s)
        if k == 0:
            before = used_bytes()
    # 0.4 GB of slots each; their other arrays are some 20 MB
    assert used_bytes() - before <= 7 * (64 << 20)
    first = systems[0].get_rates()
    for s in systems[::-1]:
        s.solve()
        assert np.array_equal(s.get_rates(), first)
        s.close()
    assert used_bytes() < before  # the last one gives the slots back


def test_a_captured_step_follows_its_slots(own):
    """Graph replays before and after a larger plan has moved the shared slots."""
    def run(larger):
        s = System(own, [3000], 1e-3, "f32")
        s.set_particles(*particles(3000, 7))
        s.rk4(0.005, 2, use_graph=True)
        if larger:
            t = System(own, [20000], 1e-3, "f32")
            t.set_particles(*particles(20000, 8))
            t.solve()
        s.rk4(0.005, 2, use_graph=True)
        out = s.get_states()
        s.close()
        if larger:
            t.close()
        return out
    assert np.array_equal(run(False), run(True))


def filled(leave):
    """Takes all device memory but about `leave` bytes."""
    torch.cuda.empty_cache()
    filler = []
    while torch.cuda.mem_get_info()[0] > leave + (32 << 20):
        filler.append(torch.empty(torch.cuda.mem_get_info()[0] - leave >> 21 << 21, dtype=torch.uint8, device="cuda"))
    return filler


@pytest.mark.parametrize("n,prec", [(32768, "f32"), (32768, "f64"), (65536, "f32")])
def test_a_full_device_takes_smaller_phases(own, n, prec):
    """128 MB left on the device: the slots (403 MB) in phases of as many rows as fit."""
    a = particles(n, 10)
    rates = []
    for full in (False, True):
        s = System(own, [n], 1e-3, prec)
        filler = filled(128 << 20) if full else []
        try:
            s.set_particles(*a)
            s.rk4(0.005, 1, use_graph=True)
            s.set_states(np.concatenate([a[0].ravel(), a[1].ravel()]))
            s.solve()
            rates.append(s.get_rates())
        finally:
            del filler
            torch.cuda.empty_cache()
            s.close()
    assert rms_rel(rates[1], rates[0]) < 1e-12  # (the grouping of the FP64 sums)


@pytest.mark.parametrize("batched", [False, True])
def test_autotune_passes_over_what_does_not_fit(own, batched):
    """128 MB left on the device: the symmetric engine's slots (403 MB) do not fit,
    a one-sided tiling's partial sums do."""
    a = particles(32768, 9)
    s = System(own, [32768], 1e-3, "f32")
    s.set_config(128, unroll=4, items_per_slot=4)  # one-sided
    s.set_particles(*a)
    s.solve()
    want = s.get_rates()
    b = Batch(own, [s])
    b.set_config(128, unroll=4, items_per_slot=4)
    b.solve()
    filler = filled(128 << 20)
    try:
        (b if batched else s).autotune()
        (b if batched else s).solve()
        got = s.get_rates()
    finally:
        del filler
        torch.cuda.empty_cache()
    assert rms_rel(got, want) <= TOL_F32_RMS
    b.close()
    s.close()


def test_a_served_request_in_phases_of_single_tiles(own):
    """32,768 particles: 403 MB of slots, above the serving engine's bound, in two
    phases."""
    sc = g.ring_pair(n_stations=2048, seed=11, nu=1e-3, steps=1)
    srv = Server(own, budget_bytes=8 << 30)
    rid = srv.submit_scenario(sc)[1]
    assert srv.wait(rid, 120)
    out = srv.fetch(rid)[0]
    srv.close()
    solo = System.from_scenario(own, sc, "f32")
    solo.rk4(sc.dt, sc.steps)
    st0 = sc.state()
    assert rms_rel(out - st0, solo.get_states() - st0) < 1e-12
    solo.close()
