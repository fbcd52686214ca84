"""The O(N^2) diagnostics at the edges of their decomposition: two particles,
one tile less and more than 128, ranges that do not divide the system, several
wakes (the kinetic energy counts pairs inside a wake twice)."""
import numpy as np
import pytest

import oracle
from pawan_b200 import System
from pawan_b200 import geometry as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 127, 128, 129, 1000, 4097, 9001])
def test_quadratic_diagnostics_against_restatement(ctx, n):
    sc = g.helical_wake(n_stations=-(-n // 32), seed=n, turns=2.0)
    pos, vor, rad, vol = (a[:n].copy() for a in sc.union())
    rad *= np.random.default_rng(n).uniform(0.7, 1.3, n)
    counts = [n // 3, n - n // 3] if n >= 3 else [1, 1]
    s = System(ctx, counts, 0.0, "f32")
    s.set_particles(pos, vor, rad, vol)
    d = s.diagnose()
    wid = np.repeat([0, 1], counts).astype(np.int32)
    # FP64 sums of the same terms: rounding of at most a few ulp of each sum's
    # magnitude; the helicity's terms cancel against the enstrophy's scale
    assert abs(d["enstrophy"] / oracle.enstrophy(pos, vor, rad) - 1) < 1e-12
    assert abs(d["helicity"] - oracle.helicity(pos, vor, rad)) < 1e-10 * abs(d["enstrophy"])
    assert abs(s.kinetic_energy() / oracle.kinetic_energy(wid, pos, vor, rad) - 1) < 1e-12
    again = s.diagnose()
    assert again["enstrophy"] == d["enstrophy"] and again["helicity"] == d["helicity"]
