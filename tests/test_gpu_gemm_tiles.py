"""FP64 tiled products on both sides of the size at which they take 64 x 64 tiles, through the blocked LU
inverse, whose trailing updates shrink across it."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(1100, 1), (1600, 1), (1700, 1), (700, 6)])
def test_blocked_inverse(n, batch):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import __graft_entry__
    __graft_entry__.build()
    from khepri_gb300 import _capi
    lib = _capi.load()
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(batch, n, n, dtype=torch.complex128, device="cuda", generator=g)
    A += 0.5 * n ** 0.5 * torch.eye(n, device="cuda")
    a, x = A.clone(), torch.empty_like(A)
    st = torch.zeros(batch, dtype=torch.int32, device="cuda")
    ws = torch.empty(lib.khp_inverse_workspace(batch, n), dtype=torch.uint8, device="cuda")
    _capi.check(lib.khp_inverse(batch, n, 0, _capi.ptr(a), n * n, _capi.ptr(x), n * n, _capi.ptr(st), _capi.ptr(ws),
                                ws.numel(), _capi.stream_ptr()), "khp_inverse")
    assert not st.any()
    resid = (A @ x - torch.eye(n, device="cuda")).abs().amax(dim=(1, 2))
    cond = torch.linalg.cond(A)
    assert (resid <= 8 * n * 2.0 ** -52 * cond).all()  # normwise bound of the inverse
