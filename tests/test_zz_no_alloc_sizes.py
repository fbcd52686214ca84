"""pawan_interact_noalloc where its decomposition changes: 2 to 4 threads per
target at 4,096 particles, the most source chunks that the fixed array holds
(5,633 and 16,383: a ragged last chunk), ragged tiles."""
import numpy as np
import pytest
import torch

import oracle
from pawan_b200 import geometry as g
from helpers import TOL_F32_MAX, TOL_F32_RMS, max_rel, rms_rel
from test_zz_no_alloc import run_noalloc

pytestmark = pytest.mark.gpu


class Cut:
    """A ring pair cut to n particles."""

    def __init__(self, n):
        sc = g.ring_pair(n_stations=-(-n // 16), seed=n, nu=1e-3)
        self.n, self.nu = n, 1e-3
        self.arrays = tuple(a[:n].copy() for a in sc.union())

    def union(self):
        return self.arrays


@pytest.mark.parametrize("n", [2, 33, 127, 128, 129, 1537, 4096, 4097, 5633, 16383])
def test_sizes_against_restatement(n):
    sc = Cut(n)
    u, da = run_noalloc(sc)
    t = np.arange(n) if n <= 512 else np.unique(np.concatenate(
        [[0, n - 1], np.random.default_rng(n).choice(n, 254, replace=False)]))
    u_ref, da_ref = oracle.pairs(*sc.union(), sc.nu, targets=t)
    assert rms_rel(u[t], u_ref) <= TOL_F32_RMS and max_rel(u[t], u_ref) <= TOL_F32_MAX
    assert rms_rel(da[t], da_ref) <= TOL_F32_RMS and max_rel(da[t], da_ref) <= TOL_F32_MAX
    # the counters are ready for the next call
    u2, da2 = run_noalloc(sc)
    assert np.array_equal(u, u2) and np.array_equal(da, da2)
