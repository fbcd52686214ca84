"""States and rates to the caller's memory, at the edges of the staged copies (one
lane up to 128 KB, four up to 1 MB, direct beyond): byte for byte."""
import numpy as np
import pytest
import torch

from pawan_b200 import System

pytestmark = pytest.mark.gpu

# bytes of a state: 48 per particle; of one wake's rates the same
EDGES = [[5], [2730], [2731], [17, 2713], [17, 1, 2713], [21845], [21846], [9000, 1, 12844], [30000, 7, 21846]]


@pytest.mark.parametrize("counts", EDGES, ids=lambda c: "+".join(map(str, c)))
def test_states_round_trip_and_rates_agree(ctx, counts):
    n = sum(counts)
    rng = np.random.default_rng(n)
    s = System(ctx, counts, 1e-3, "f32")
    s.set_particles(rng.uniform(-1, 1, (n, 3)), rng.normal(size=(n, 3)), np.full(n, 0.1), np.full(n, 1e-3))
    for seed in (1, 2):
        state = np.random.default_rng(seed).uniform(-1, 1, 6 * n)
        s.set_states(state)
        assert np.array_equal(s.get_states(), state)
    s.solve()
    rates = s.get_rates()
    pinned = torch.empty(6 * n, dtype=torch.float64, pin_memory=True).numpy()
    assert np.array_equal(s.get_rates(out=pinned), rates)
    o = 0
    for w, c in enumerate(counts):
        u, da = s.wake_rates(w)
        assert np.array_equal(np.concatenate([u.ravel(), da.ravel()]), rates[6 * o:6 * (o + c)])
        o += c
    s.close()
