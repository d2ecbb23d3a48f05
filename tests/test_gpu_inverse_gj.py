"""Batched explicit inverse by Gauss-Jordan elimination (khp_inverse_gj) against numpy's inverse: FP32
sizes on both sides of every register tile and of the change to row panels, both precisions on both
sides of a panel, of a block of update tiles and of the one-thread-per-column limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import __graft_entry__
    __graft_entry__.build()
    from khepri_gb300 import _capi
    return _capi.load()


def _inverse(lib, A, precision):
    import torch
    from khepri_gb300 import _capi
    batch, n, _ = A.shape
    dt = torch.complex128 if precision == 0 else torch.complex64
    a = torch.from_numpy(A).to(dt).cuda().contiguous()
    x = torch.empty_like(a)
    st = torch.zeros(batch, dtype=torch.int32, device="cuda")
    ws = torch.empty(lib.khp_inverse_workspace(batch, n), dtype=torch.uint8, device="cuda")
    _capi.check(lib.khp_inverse_gj(batch, n, precision, _capi.ptr(a), n * n, _capi.ptr(x), n * n, _capi.ptr(st),
                                   _capi.ptr(ws), ws.numel(), _capi.stream_ptr()), "khp_inverse_gj")
    torch.cuda.synchronize()
    return x.cpu().numpy().astype(np.complex128), st.cpu().numpy()


@pytest.mark.parametrize("precision,n", [(1, n) for n in (1, 2, 31, 32, 33, 56, 57, 64, 65, 80, 81, 96, 97, 112, 113,
                                                          128, 129, 160, 161, 192, 242, 513, 1024, 1025)]
                         + [(0, n) for n in (1, 7, 8, 9, 32, 33, 64, 65, 100, 242, 520, 1024)])
def test_matches_numpy_inverse(lib, precision, n):
    rng = np.random.default_rng(1000 + n)
    batch = 3 if n < 500 else 1
    A = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    A += 0.5 * np.sqrt(n) * np.eye(n)  # moderately conditioned, pivoting still active
    if precision == 1:
        A = A.astype(np.complex64).astype(np.complex128)
    X, st = _inverse(lib, A, precision)
    assert (st == 0).all()
    ref = np.linalg.inv(A)
    # normwise bound: |X - inv(A)| <= c n eps cond(A) |inv(A)|
    eps = 2.0 ** -52 if precision == 0 else 2.0 ** -23
    cond = np.linalg.cond(A)
    err = np.abs(X - ref).max(axis=(1, 2)) / np.abs(ref).max(axis=(1, 2))
    assert (err <= 8 * n * eps * cond).all(), (err, cond)
    assert np.abs(A @ X - np.eye(n)).max() <= 8 * n * eps * cond.max()


@pytest.mark.parametrize("precision,n", [(1, 40), (1, 100), (1, 150), (0, 64)])
def test_pivoting_and_status(lib, precision, n):
    rng = np.random.default_rng(7)
    base = np.triu(rng.standard_normal((n, n))) * 0.1 + 4 * np.eye(n) + 0j
    A = np.stack([base[rng.permutation(n)] for _ in range(4)])  # zero leading entries: every step must pivot
    good = A[0].copy()
    A[1, :, 5] = 0.0        # a zero column: singular
    A[2, 7, :] = 0.0        # a zero row: singular
    A[3, 3, 3] = np.nan     # a NaN
    X, st = _inverse(lib, A, precision)
    assert st[0] == 0
    tol = 1e-10 if precision == 0 else 1e-3
    assert np.abs(good @ X[0] - np.eye(n)).max() < tol
    assert st[1] & 1 and st[2] & 1 and st[3] & 4
