"""The packed backward passes of the 16-bit collision (psl_collision_g.cuh), compiled for the
host: each half of a pair is the scalar pass's result, bit for bit."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def passes():
    gxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    build = os.path.join(REPO, "tests", "_build")
    os.makedirs(build, exist_ok=True)
    so = os.path.join(build, "collision_g_pairs_host.so")
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(REPO, "periodicshiftlbm_b200", "csrc"),
                    os.path.join(REPO, "tests", "native", "collision_g_pairs_host.cpp"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    for name in ("passes_pair", "passes_scalar"):
        getattr(L, name).argtypes = [ctypes.c_void_p, ctypes.c_float, ctypes.c_float, ctypes.c_float, ctypes.c_int]
    for name in ("backward_pair", "backward_scalar"):
        getattr(L, name).argtypes = [ctypes.c_void_p, ctypes.c_float, ctypes.c_float, ctypes.c_void_p]
    return L


@pytest.mark.parametrize("weights", [0, 1])
def test_pair_is_two_scalar_passes(passes, weights):
    rng = np.random.default_rng(4)
    for _ in range(200):
        # (m0, m1, m2) of two lines, magnitudes as the collision's: rho and small moments
        m = np.concatenate([1.0 + rng.uniform(-0.02, 0.02, (2, 1)), rng.uniform(-0.2, 0.2, (2, 2))], 1).astype(np.float32)
        u = np.float32(rng.uniform(-0.1, 0.1))
        a, b = m.copy(), m.copy()
        passes.passes_pair(a.ctypes.data, u, 1.0 / 54.0, 2.0 / 27.0, weights)
        passes.passes_scalar(b.ctypes.data, u, 1.0 / 54.0, 2.0 / 27.0, weights)
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_both_passes_in_pairs_are_the_scalar_ones(passes):
    """Every line with its own weights and in its own slot: 27 distinct moments."""
    rng = np.random.default_rng(5)
    for _ in range(200):
        m = rng.uniform(-0.3, 0.3, 27).astype(np.float32)
        uy, uz = rng.uniform(-0.1, 0.1, 2).astype(np.float32)
        a, b = np.empty(27, np.float32), np.empty(27, np.float32)
        passes.backward_pair(m.ctypes.data, uy, uz, a.ctypes.data)
        passes.backward_scalar(m.ctypes.data, uy, uz, b.ctypes.data)
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
