"""Pieces of the per-CTA eigensolver by themselves (tests/device/eigen_probe.cu, built here with nvcc)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
EPS = np.finfo(np.float64).eps
D = ctypes.POINTER(ctypes.c_double)


def _p(a):
    return a.ctypes.data_as(D)


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("probe") / "eigen_probe.so")
    nvcc = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else "nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    "-I", os.path.join(HERE, "..", "pm3-rs_b200", "csrc"), "-o", out,
                    os.path.join(HERE, "device", "eigen_probe.cu")], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("n,kval", [(2, 2), (7, 4), (40, 23), (256, 256)])
def test_eigenvalues_to_their_own_last_bits(probe, n, kval):
    """Diagonal matrices: the counts are exact, so the search may stop no earlier than at an interval of 2 eps |lambda|, whatever
    the norm; its middle is within eps |lambda| of the value."""
    rng = np.random.default_rng(n)
    d = rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-9.0, 2.0, n)
    d[0], d[-1] = 150.0, -1.0e-8
    lam = np.zeros(kval)
    assert probe.probe_eigenvalues(n, kval, _p(d), _p(np.zeros(n)), _p(lam)) == 0
    want = np.sort(d)[:kval]
    assert (np.abs(lam - want) <= 2 * EPS * np.abs(want)).all()


def test_root_and_reciprocal_of_the_reflectors(probe):
    """Newton-Raphson from a 20-bit approximation: the last step's fma rounds a value whose error is far below an ulp, so the
    results are the neighbours of the exact ones and within one unit of CUDA's correctly rounded functions."""
    worst = (ctypes.c_ulonglong * 2)()
    assert probe.probe_roots(20000, worst) == 0
    assert worst[0] <= 1 and worst[1] <= 1, list(worst)
