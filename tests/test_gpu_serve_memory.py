"""What a serving budget admits: requests that fit with one-sided partial sums of
8,192-source chunks beside their arrays are accepted, and as many at a time, although
the symmetric engine's slots alone are larger than that."""
import time

import numpy as np
import pytest

from pawan_b200 import Server, System
from pawan_b200 import geometry as g
from helpers import TOL_F32_RMS, rms_rel

pytestmark = pytest.mark.gpu


def one_sided_bytes(n, prec):
    """Arrays and rates, partial sums of each chunk (FP32: near ones too)."""
    chunks = -(-n // 8192)
    partial = 48.0 * (n + 512) * chunks if chunks > 1 else 0.0
    near = 49.0 * (n + 512) * chunks if prec == "f32" else 0.0
    return 437.0 * n + 4096.0 + partial + near


@pytest.mark.parametrize("n", [2048, 8192, 32768, 66560])
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_a_request_that_fits_is_served(ctx, n, prec):
    sc = g.ring_pair(n_stations=n // 16, seed=21, nu=1e-3, steps=1)
    srv = Server(ctx, budget_bytes=one_sided_bytes(n, prec), precision=prec)
    status, rid = srv.submit_scenario(sc)
    assert status == 0
    assert srv.wait(rid, 120)
    out = srv.fetch(rid)[0]
    assert srv.stats()["bytes_in_use"] == 0
    srv.close()
    solo = System.from_scenario(ctx, sc, prec)
    solo.rk4(sc.dt, sc.steps)
    st0 = sc.state()
    assert rms_rel(out - st0, solo.get_states() - st0) < (TOL_F32_RMS if prec == "f32" else 1e-12)
    solo.close()


# (of 8,192 particles, whose arrays are nearly all of it, nine of ten)
@pytest.mark.parametrize("n,prec,least", [(8192, "f32", 9), (32768, "f32", 10), (16384, "f64", 9)])
def test_as_many_at_a_time(ctx, n, prec, least):
    """A budget of ten: they are admitted together, and finish as they do alone."""
    sc = g.ring_pair(n_stations=n // 16, seed=22, nu=1e-3, steps=1)
    srv = Server(ctx, budget_bytes=10 * one_sided_bytes(n, prec), precision=prec)
    ids = [srv.submit_scenario(sc, nsteps=10_000_000)[1] for _ in range(10)]
    most, deadline = 0, time.time() + 15
    while most < least and time.time() < deadline:
        most = max(most, srv.stats()["active"])
        time.sleep(0.001)
    for rid in ids:
        srv.cancel(rid)
    for rid in ids:
        assert srv.wait(rid, 60)
    srv.close()
    assert most >= least


def test_result_does_not_depend_on_the_waves(ctx):
    """Sixteen requests whose slots (25 MB each) share a buffer of 32 MB."""
    scs = [g.ring_pair(n_stations=512, seed=30 + k, nu=1e-3, steps=2) for k in range(16)]
    states = []
    for together in (True, False):
        srv = Server(ctx, budget_bytes=256 << 20)
        ids = []
        for sc in scs:
            ids.append(srv.submit_scenario(sc)[1])
            if not together:
                assert srv.wait(ids[-1], 60)
        for rid in ids:
            assert srv.wait(rid, 60)
        states.append([srv.fetch(rid)[0] for rid in ids])
        srv.close()
    for a, b in zip(*states):
        assert np.array_equal(a, b)
