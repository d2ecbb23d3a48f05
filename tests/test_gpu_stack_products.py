"""The matrix-vector products of the stack refinement and of its adjoint, at sizes below, at and above
one and two warps of rows and on both sides of the batch at which a problem's kernels take 512 threads:
totals and the gradient of the zeroth transmitted order against autograd of the complex128 restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pw", [(1, 1), (1, 3), (5, 3), (3, 11), (7, 7)])  # n = 2, 6, 30, 66, 98
@pytest.mark.parametrize("copies", [1, 153])  # 2 and 306 problems
def test_totals_and_gradient(pw, copies):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import __graft_entry__
    __graft_entry__.build()
    from khepri_gb300 import autograd, workloads
    from oracle import torch_c128 as tc
    m = np.asarray(workloads.disc_canvas(32, 0.3, 3.0, 1.5), np.float64)
    m = m + 0.2 * np.sin(np.arange(m.size)).reshape(m.shape)
    stack = ["A", "U", "B"]
    wl = np.array([1.31, 1.73])
    c = (pw[0] * pw[1] - 1) // 2
    eps = torch.tensor(m[None], dtype=torch.float64, device="cuda", requires_grad=True)
    structs = [(pw, {"A": ("pixmap", 0, 0.3), "B": ("pixmap", 0, 0.3), "U": ("uniform", 2.1, 0.6)}, stack)]
    out = autograd.solve_rt(eps, structs, np.tile(wl, copies), np.zeros((2 * copies, 2)),
                            which=np.zeros(2 * copies, np.int64))
    assert not out[-1].any()
    out[3][:, c].mean().backward()
    e = torch.tensor(m, dtype=torch.float64, requires_grad=True)
    lay = {"A": ("pixmap", e, 0.3), "B": ("pixmap", e, 0.3), "U": ("uniform", 2.1, 0.6)}
    ref = torch.stack([tc.solve_orders(pw, lay, stack, w)[3][c] for w in wl])
    if pw == (1, 1):  # exactly degenerate modes, where autograd of eig is undefined: T depends on the mean
        d = [np.mean([tc.solve_orders(pw, {"A": ("pixmap", e.detach() + h, 0.3), "B": ("pixmap", e.detach() + h, 0.3),
                                                "U": lay["U"]}, stack, w)[3][c].item()
                      for w in wl]) for h in (1e-5, -1e-5)]
        gr = np.full(m.shape, (d[0] - d[1]) / 2e-5 / m.size)
    else:
        ref.mean().backward()
        gr = e.grad.numpy()
    t0 = out[3][:, c].detach().cpu().numpy().reshape(copies, 2)
    # FP64 results of well-conditioned stacks; the adjoint's FP32 products leave 2e-6 of the largest
    # component per pixel (x 5)
    np.testing.assert_allclose(t0, np.broadcast_to(ref.detach().numpy(), t0.shape), rtol=0, atol=1e-9)
    g = eps.grad[0].cpu().numpy()
    assert np.abs(g - gr).max() <= 1e-5 * np.abs(gr).max()
