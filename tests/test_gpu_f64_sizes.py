"""The tuned FP64 pairs at the edges of the symmetric engine's decomposition:
a few particles, one tile less and more than 128, the largest system in single
tile pairs (256 tiles) and the smallest in groups, both smoothing kernels."""
import numpy as np
import pytest

import oracle
from pawan_b200 import System
from helpers import TOL_F64T_MAX, TOL_F64T_RMS, max_rel, rms_rel
from test_gpu_symmetric import EDGE, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["highorder", "gaussian"])
@pytest.mark.parametrize("n", [3, 33, 127, 129, 1000, EDGE, EDGE + 1])
def test_f64_against_restatement(ctx, n, kernel):
    arrays = particles(n, mixed=True)
    t = np.arange(n) if n <= 512 else np.unique(np.concatenate(
        [[0, n - 1], np.random.default_rng(n).choice(n, 126, replace=False)]))
    s = System(ctx, [n], 0.0, "f64")
    s.set_kernel(kernel)
    s.set_particles(*arrays)
    for nu in (0.0, 1e-3):
        s.set_nu(nu)
        s.solve()
        u, da = s.union_rates()
        u_ref, da_ref = oracle.pairs(*arrays, nu, targets=t, kernel=kernel)
        assert rms_rel(u[t], u_ref) <= TOL_F64T_RMS and max_rel(u[t], u_ref) <= TOL_F64T_MAX
        assert rms_rel(da[t], da_ref) <= TOL_F64T_RMS and max_rel(da[t], da_ref) <= TOL_F64T_MAX
