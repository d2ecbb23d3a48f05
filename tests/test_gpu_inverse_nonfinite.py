"""Infinite entries in the batched Gauss-Jordan inverse: the matrix is flagged as non-finite wherever the
entry stands (as the pivot of its row or beside it) and its neighbours in the batch are not; sizes of
the register form and of the panel form.  khp_structure_prep, which inverts convolution matrices, too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
PLACES = [(0, 0), (1, 2), (2, 0), (-1, -1), (-1, 0), (0, -1)]
VALUES = [np.inf, -np.inf, complex(0, np.inf)]


@pytest.fixture(scope="module")
def lib():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import __graft_entry__
    __graft_entry__.build()
    from khepri_gb300 import _capi
    return _capi.load()


def _matrices(n):
    """One finite matrix between every two with an infinite entry."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((2 * len(PLACES) * len(VALUES), n, n)) + 3 * np.eye(n) + 0j
    bad = [(p, v) for p in PLACES for v in VALUES]
    for i, ((r, c), v) in enumerate(bad):
        A[2 * i, r, c] = v
    return A


def _check(status):
    assert (status[::2] & 4).all() and not status[1::2].any()


@pytest.mark.parametrize("precision,n", [(1, 4), (1, 25), (1, 60), (1, 128), (1, 129), (1, 160), (0, 4), (0, 9),
                                         (0, 25), (0, 49), (0, 81)])
def test_infinite_entry_is_flagged(lib, precision, n):
    import torch
    from khepri_gb300 import _capi
    a = torch.from_numpy(_matrices(n)).to(torch.complex128 if precision == 0 else torch.complex64).cuda()
    x, st = torch.empty_like(a), torch.zeros(len(a), dtype=torch.int32, device="cuda")
    ws = torch.empty(lib.khp_inverse_workspace(len(a), n), dtype=torch.uint8, device="cuda")
    _capi.check(lib.khp_inverse_gj(len(a), n, precision, _capi.ptr(a), n * n, _capi.ptr(x), n * n, _capi.ptr(st),
                                   _capi.ptr(ws), ws.numel(), _capi.stream_ptr()), "khp_inverse_gj")
    _check(st.cpu().numpy())


@pytest.mark.parametrize("nh", [4, 9, 25])
def test_infinite_convolution_matrix_is_flagged(lib, nh):
    import torch
    from khepri_gb300 import _capi
    c = torch.from_numpy(_matrices(nh)).cuda()
    ic, hx, hy = (torch.empty_like(c) for _ in range(3))
    g = torch.linspace(-3, 3, nh, dtype=torch.float64, device="cuda")
    st = torch.zeros(len(c), dtype=torch.int32, device="cuda")
    ws = torch.empty(lib.khp_structure_prep_workspace(len(c), nh), dtype=torch.uint8, device="cuda")
    _capi.check(lib.khp_structure_prep(len(c), nh, _capi.ptr(c), _capi.ptr(g), _capi.ptr(g), _capi.ptr(ic),
                                       _capi.ptr(hx), _capi.ptr(hy), _capi.ptr(st), _capi.ptr(ws), ws.numel(),
                                       _capi.stream_ptr()), "khp_structure_prep")
    _check(st.cpu().numpy())
