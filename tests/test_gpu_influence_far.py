"""Vorticity field of particles so far apart that the squared distance is not a
double: those pairs contribute nothing, and the others what they always do."""
import numpy as np
import pytest

from pawan_b200 import System

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["highorder", "gaussian"])
@pytest.mark.parametrize("n", [6, 300])
def test_field_across_an_overflowing_distance(ctx, n, kernel):
    rng = np.random.default_rng(n)
    pos, vor = rng.uniform(-1, 1, (n, 3)), rng.normal(size=(n, 3))
    rad, vol = np.full(n, 0.3), np.full(n, 1e-3)
    far = pos.copy()
    far[n // 2:, 0] = 1e200  # (on one another along x: their y and z stay apart)
    fields = []
    for p in (pos[: n // 2], far):
        s = System(ctx, [len(p)], 0.0, "f64")
        s.set_kernel(kernel)
        s.set_particles(p, vor[: len(p)], rad[: len(p)], vol[: len(p)])
        cols = s.influence_columns(np.stack([vor[: len(p)]] * 2))
        fields.append(s.influence())
        assert np.array_equal(cols[0], fields[-1]) and np.array_equal(cols[1], fields[-1])
        s.close()
    near, both = fields
    assert np.isfinite(both).all()
    # the same terms, in chunks of another length: |terms| add up to at most Z(0) sum |alpha|
    total = 1.875 / np.pi / 0.3 ** 3 * np.abs(vor[: n // 2]).sum()
    assert np.abs(both[: n // 2] - near).max() <= n * 2.0 ** -52 * total
