"""The vorticity field where its decomposition changes: source chunks that a
system's size sets (one from 32,768 particles on), tiles of 64 and 128 targets,
column groups (32 columns) and register tiles of two columns."""
import math

import numpy as np
import pytest

from pawan_b200 import System
from helpers import TOL_F64_MAX, TOL_F64_RMS, max_rel, rms_rel

pytestmark = pytest.mark.gpu


def field_at(t, pos, rad, alpha):
    """Z alpha at the targets t, in numpy."""
    out = np.empty((t.size, 3))
    for k, i in enumerate(t):
        r2 = ((pos[i] - pos) ** 2).sum(1)
        s2 = 0.5 * (rad[i] ** 2 + rad ** 2)
        out[k] = (1.875 / math.pi * (r2 / s2 + 1.0) ** -7.5 / s2 ** 1.5) @ alpha
    return out


@pytest.mark.parametrize("n,columns", [(2, 1), (33, 2), (65, 3), (1000, 33), (4097, 65), (32767, 2), (32769, 3)])
def test_field_and_columns(ctx, n, columns):
    rng = np.random.default_rng(n)
    pos = rng.uniform(-1, 1, (n, 3))
    rad = rng.uniform(0.05, 0.2, n)
    alpha = rng.standard_normal((columns, n, 3))
    s = System(ctx, [n], 0.0, "f32")
    s.set_particles(pos, alpha[-1], rad, np.full(n, 1e-4))
    k = s.influence_columns(alpha)
    assert np.array_equal(k[-1], s.influence())
    t = np.unique(np.concatenate([[0, n - 1], rng.choice(n, min(n, 64), replace=False)]))
    for c in (0, columns // 2, columns - 1):
        ref = field_at(t, pos, rad, alpha[c])
        assert rms_rel(k[c][t], ref) <= TOL_F64_RMS and max_rel(k[c][t], ref) <= TOL_F64_MAX
    # the kept scratch serves a smaller and then the same request again
    assert np.array_equal(s.influence_columns(alpha[:1])[0], k[0])
    assert np.array_equal(s.influence_columns(alpha), k)
