"""The FP64 1/sqrt of the pair kernels (rsqrt64.cuh) against extended precision
and CUDA's own function, over the whole range of normal doubles.

Bound: the estimate is good to 2^-19 (20 bits and a cut-off argument), so the
iteration's 5/16 e^3 and its small roundings stay below 0.03 units in the last
place, and the last operation rounds once: 0.53.  CUDA's is documented to 1."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("rsqrt64") / "librsqrt64.so")
    r = subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                        "-I" + os.path.join(ROOT, "pawan_b200", "csrc"), "-shared", "-Xcompiler", "-fPIC",
                        os.path.join(ROOT, "tests", "abi", "rsqrt64.cu"), "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(so)

    def call(x):
        t = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        out = torch.zeros((3, len(x)), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert lib.rsqrt64_probe(ctypes.c_void_p(t.data_ptr()), ctypes.c_void_p(out.data_ptr()), len(x)) == 0
        return out.cpu().numpy()
    return call


@pytest.mark.parametrize("lo,hi", [(0, 2), (-40, 40), (-1022, 1024)])
def test_error_in_units_of_the_last_place(probe, lo, hi):
    x = 2.0 ** np.random.default_rng(hi).uniform(lo, hi, 1 << 20)
    x = x[np.isfinite(x) & (x >= np.finfo(float).tiny)]
    own, full, cuda = probe(x)
    exact = 1 / np.sqrt(x.astype(np.longdouble))
    ulp = np.spacing(exact.astype(np.float64))
    assert np.abs((own - exact) / ulp).max() <= 0.53
    assert np.array_equal(own, full)
    assert np.abs((own - cuda) / ulp).max() <= 1.0


def test_values_outside_the_normal_range(probe):
    tiny = np.finfo(float).tiny
    x = np.array([0.0, tiny / 8, np.inf, np.nan, -1.0, tiny, np.finfo(float).max])
    own, full, cuda = probe(x)
    assert np.isnan(own[[0, 2, 3, 4]]).all() and own[1] == np.inf
    assert full[0] == np.inf and full[1] == np.inf and full[2] == 0.0 and np.isnan(full[3:5]).all()
    assert np.array_equal(full[[0, 2, 5, 6]], cuda[[0, 2, 5, 6]])
