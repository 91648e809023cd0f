"""The FP64 pair kernels' reciprocal square root against 80-bit values and
CUDA's rsqrt over the normal range, and the Barnes-Hut sums where a squared
distance leaves it: a finite particle so far away that r^2 overflows adds
nothing, as its 1 / r^2 does."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle_lib as O
from conftest import E, ROOT, gaussian_cloud

pytestmark = pytest.mark.gpu


def test_rsqrt_over_the_normal_range(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    so = str(tmp_path / "librsqrt.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", f"-I{ROOT}/include", f"-I{ROOT}/antimatter-kernel_b200/csrc",
                    os.path.join(ROOT, "tests", "rsqrt_harness.cu"), "-o", so], check=True, capture_output=True)
    rng = np.random.default_rng(3)
    eps = np.finfo(float).eps
    # mantissas at both ends of an octave and inside it, in every normal octave
    m = np.concatenate([[1.0, 1.0 + eps, 1.0 + 2 * eps, 1.5, 2.0 - eps, 2.0 - 2 * eps], 1.0 + rng.random(250)])
    x = np.ldexp(m[None, :], np.arange(-1022, 1024)[:, None]).ravel()
    assert np.all(np.isfinite(x)) and x.min() == np.finfo(float).tiny and x.max() == np.finfo(float).max
    own, cuda = np.empty_like(x), np.empty_like(x)
    p = [a.ctypes.data_as(C.POINTER(C.c_double)) for a in (x, own, cuda)]
    assert C.CDLL(so).rsqrt_run(len(x), *p) == 0
    exact = 1.0 / np.sqrt(x.astype(np.longdouble))
    ulp = np.spacing(exact.astype(float)).astype(np.longdouble)
    assert np.max(np.abs(own - exact) / ulp) <= 2.0
    assert np.max(np.abs(own - cuda) / ulp) <= 3.0  # CUDA's rsqrt is within 1 ulp of the value


@pytest.mark.parametrize("far", [1e100, 1.2e154, 1.5e154, 1e160, 1e300])
@pytest.mark.parametrize("theta", [0.0, 0.5])
def test_barnes_hut_with_a_far_particle(sim, far, theta):
    # the tree's depth limit keeps the cloud in one leaf: the exact sums
    x, y, z, q = gaussian_cloud(900, 7)
    x[0], y[0], z[0], q[0] = far, -0.5 * far, 0.25 * far, E
    got = sim.solve_barnes_hut(x, y, z, q, theta, want_phi=True)
    ref = O.allpairs(x, y, z, q, want_phi=True)
    for a, b in zip(got, ref):
        assert np.all(np.isfinite(a))
        assert np.max(np.abs(a - b)) <= 1e-10 * np.max(np.abs(b))
