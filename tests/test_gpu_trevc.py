"""Eigenvectors of the FP64 eigensolver through the pencil of random S-matrices, at sizes below, at and
above one and two blocks of rows and of columns, and on both sides of the largest size whose columns are
solved by themselves; two matrices per call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [2, 4, 8, 10, 14, 16, 18, 24, 34, 212, 214])
def test_eigenvectors_of_random_pencils(khp, h):
    from khepri_gb300 import eigentricks as et
    rng = np.random.default_rng(h)
    S = (rng.standard_normal((2, 2 * h, 2 * h)) + 1j * rng.standard_normal((2, 2 * h, 2 * h))) / np.sqrt(2 * h)
    w, v = et.scattering_eigenvalues(S)
    for i in range(2):
        Sl, Sr = et.scattering_splitlr(S[i])
        # backward error n eps of the standard problem, times the condition of Sr (random: ~ n)
        tol = 1e-15 * (2 * h) ** 2 * np.linalg.cond(Sr)
        scale = np.abs(Sl).max() + np.abs(Sr).max() * np.abs(w[i])
        assert (np.abs(Sl @ v[i] - (Sr @ v[i]) * w[i]) / scale).max() < max(tol, 1e-13)
        assert np.allclose(np.linalg.norm(v[i], axis=0), 1.0)
