"""Convolution matrices against numpy's FFT, at canvas sizes below, at and above the block's groups of x,
its chunk of x, its table of roots and its largest number of columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 1), (17, 5), (64, 64), (5, 171), (33, 256), (512, 257), (513, 511), (9, 512),
                                   (1025, 513), (31, 1024), (30, 1025), (7, 8192)])
@pytest.mark.parametrize("nmaps", [1, 3])
def test_convmat_matches_fft(nx, ny, nmaps):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import __graft_entry__
    __graft_entry__.build()
    from khepri_gb300 import _capi, engine
    lib = _capi.load()
    px = min(5, (nx + 1) // 2 - 1 + (nx + 1) // 2 % 2)
    py = min(9, (ny + 1) // 2 - 1 + (ny + 1) // 2 % 2)
    rng = np.random.default_rng(nx * 10007 + ny)
    m = rng.uniform(1, 5, (nmaps, nx, ny)) + 1j * rng.uniform(0, 1, (nmaps, nx, ny))
    eps = torch.tensor(m, dtype=torch.complex128, device="cuda")
    nh = px * py
    conv = torch.empty((nmaps, nh, nh), dtype=torch.complex128, device="cuda")
    ws = engine.workspace(lib.khp_convmat_workspace(nmaps, px, py), "cuda")
    assert lib.khp_convmat(nmaps, nx, ny, _capi.ptr(eps), px, py, _capi.ptr(conv), _capi.ptr(ws), ws.numel(),
                           _capi.stream_ptr()) == 0
    f = np.fft.fft2(m) / (nx * ny)
    h = np.arange(nh)
    p, q = h % px, h // px
    ref = f[:, (p[:, None] - p[None, :]) % nx, (q[:, None] - q[None, :]) % ny]
    # each coefficient is a mean of entries below 6; sums of at most 1025 + 8192 roundings, far from aligned
    assert np.abs(conv.cpu().numpy() - ref).max() < 6e-14
