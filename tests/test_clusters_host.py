"""Labels of the eigenvalue clusters (khp_clusters.cuh, compiled for the host): connected components of
the close eigenvalues, whatever their order.  A column whose label is not its own component's smallest index
would leave the members and the transform that its correction reads unwritten."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest
from scipy.sparse.csgraph import connected_components

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TOL, MOST, LEVELS = 1e-3, 12, 4


@pytest.fixture(scope="module")
def labels(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("needs g++")
    out = tmp_path_factory.mktemp("clustershost") / "libclusters.so"
    subprocess.run([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "khepri_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "host", "clusters_host.cpp"), "-o", str(out)], check=True)
    f = ctypes.CDLL(str(out)).host_cluster_labels

    def run(mu, fp32):
        mu = np.ascontiguousarray(mu, dtype=np.complex128)
        lb, sz = np.empty(len(mu), np.int32), np.empty(len(mu), np.int32)
        f(len(mu), mu.ctypes.data_as(ctypes.c_void_p), fp32, lb.ctypes.data_as(ctypes.c_void_p),
          sz.ctypes.data_as(ctypes.c_void_p))
        return lb, sz

    return run


def _expected(mu):
    n, tol = len(mu), TOL * np.abs(mu).max()
    lb, sz = np.arange(n), np.full(n, n + MOST)
    for _ in range(LEVELS):
        act = sz > MOST
        if not act.any():
            break
        idx = np.flatnonzero(act)
        c = connected_components(np.abs(mu[idx][:, None] - mu[idx][None, :]) < tol, directed=False)[1]
        for k in range(c.max() + 1):
            w = idx[c == k]
            lb[w], sz[w] = w[0], len(w)
        tol /= 3
    return lb, sz


def _descending(n):
    """Order of a chain of n along which a label passed on by index moves one column a round: its head, then
    the others from the last one back."""
    return np.r_[0, np.arange(n - 1, 0, -1)]


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 12, 13, 64, 65, 66, 130, 600])
@pytest.mark.parametrize("spacing", [0.9 * TOL, 0.9 * TOL / 3, 0.9 * TOL / 27])
@pytest.mark.parametrize("order", ["up", "down", "random"])
def test_chains(labels, n, spacing, order, fp32):
    pos = {"up": np.arange(n), "down": np.argsort(_descending(n)),
           "random": np.random.default_rng(n).permutation(n)}[order]
    mu = 1.0 - spacing * pos + 0j  # largest magnitude 1; 600 x 9e-4 stays within it
    lb, sz = labels(mu, fp32)
    elb, esz = _expected(mu)
    assert np.array_equal(lb, elb) and np.array_equal(sz, esz)


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("seed", range(6))
def test_dense_spectra(labels, seed, fp32):
    rng = np.random.default_rng(seed)
    n = int(rng.integers(100, 700))
    mu = -rng.uniform(0, 1, n) + 1j * rng.choice([0.0, 2e-4, 2e-2]) * rng.standard_normal(n)
    lb, sz = labels(mu, fp32)
    elb, esz = _expected(mu)
    assert np.array_equal(lb, elb) and np.array_equal(sz, esz)
    assert np.array_equal(lb[lb], lb)
