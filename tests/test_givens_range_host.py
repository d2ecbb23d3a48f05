"""FP64 QR rotations over the range of magnitudes (khp_dense.cuh for the host): matrices scaled so that the
fourth powers of their entries leave the range of FP64, matrices graded over many orders, and the
eigenpairs of ordinary ones, against the backward error c n eps of the solver."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def geev(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("needs g++")
    out = tmp_path_factory.mktemp("givenshost") / "libteamhost.so"
    subprocess.run([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "khepri_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "host", "team_dense_host.cpp"), "-o", str(out)], check=True)
    f = ctypes.CDLL(str(out)).host_geev

    def run(A):
        n = len(A)
        A = np.ascontiguousarray(A, dtype=np.complex128)
        W, lam = np.zeros_like(A), np.zeros(n, dtype=np.complex128)
        p = [a.ctypes.data_as(ctypes.c_void_p) for a in (A, W, lam)]
        assert f(n, *p) == 0
        return W, lam

    return run


def _residual(A, W, lam):
    return np.abs(A @ W - W * lam).max() / (np.abs(A).sum(axis=1).max() * np.abs(W).max())


@pytest.mark.parametrize("scale", [1e-100, 1e-75, 1e-36, 1.0, 1e36, 1e75, 1e100])
@pytest.mark.parametrize("n", [2, 17, 40])
def test_scaled(geev, n, scale):
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) * scale
    W, lam = geev(A)
    assert _residual(A / scale, W, lam / scale) <= 10 * n * 2.0 ** -52


@pytest.mark.parametrize("decades", [20, 60, 120])
def test_graded(geev, decades):
    n = 24
    rng = np.random.default_rng(decades)
    d = 10.0 ** -np.linspace(0, decades, n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) * d[:, None]
    W, lam = geev(A)
    assert np.isfinite(W).all() and _residual(A, W, lam) <= 10 * n * 2.0 ** -52
