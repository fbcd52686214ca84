"""Step sizes of a batch: a rejected call changes nothing."""
import numpy as np
import pytest

from pawan_b200 import Batch, PawanError, System
from pawan_b200 import geometry as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad_value", [-1.0, float("nan")])
@pytest.mark.parametrize("changed,bad", [(0, 2), (1, 2), (2, 0)])
def test_rejected_step_sizes_leave_no_trace(ctx, changed, bad, bad_value):
    """A call that changes one system's dt and is rejected for another's; then
    the same change with the others as they were.  The result is that of a batch
    which never saw the rejected call.  (System 1, of more than 8,192 particles,
    lies in a plan of its own.)"""
    scs = [g.single_ring(n_stations=k, seed=60 + k, nu=1e-3) for k in (40, 1030, 48)]  # N = 320, 8,240, 384
    first = np.array([0.001, 0.002, 0.003])
    second = first.copy()
    second[changed] *= 1.5
    states = []
    for rejected in (False, True):
        systems = [System.from_scenario(ctx, sc, "f32") for sc in scs]
        b = Batch(ctx, systems)
        b.rk4(first, 1)
        if rejected:
            dts = second.copy()
            dts[bad] = bad_value
            with pytest.raises(PawanError):
                b.rk4(dts, 1)
        b.rk4(second, 1)
        states.append([s.get_states() for s in systems])
    for a, c in zip(*states):
        assert np.array_equal(a, c)
