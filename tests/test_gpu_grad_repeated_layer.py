"""Gradient with respect to a layer that stands in the stack more than once: the total over its occurrences,
as for two layers of one pixmap under two names, and as torch autograd through the complex128 restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_repeated_name_counts_once(khp):
    import torch
    from khepri_gb300 import autograd, batch
    from oracle import torch_c128
    rng = np.random.default_rng(3)
    eps = 1.0 + 11.0 / (1.0 + np.exp(-rng.standard_normal((32, 32))))
    pw, f = (3, 3), np.array([0.45, 0.53])
    same = (pw, {"D": ("pixmap", eps, 0.3), "U": ("uniform", 2.1, 0.7)}, ["D", "U", "D"])
    two = (pw, {"A": ("pixmap", eps, 0.3), "B": ("pixmap", eps, 0.3), "U": ("uniform", 2.1, 0.7)}, ["A", "U", "B"])
    dT = np.zeros((2, 9))
    dT[:, 4] = 1.0
    g = [batch.solve_structures_grad([s], 1.0 / f, np.zeros((2, 2)), which=np.zeros(2, int), dT=dT)[4][0]
         for s in (same, two)]
    assert np.abs(g[0]["D"] - g[1]["A"]).max() <= 1e-12 * np.abs(g[1]["A"]).max()
    t = torch.tensor(eps, dtype=torch.float64, requires_grad=True)
    layers = {"D": ("pixmap", t, 0.3), "U": ("uniform", 2.1, 0.7)}
    sum(torch_c128.solve_orders(pw, layers, same[2], 1.0 / v)[3][4] for v in f).backward()
    ref = t.grad.numpy()
    # the contraction W H^T W^-1 of the gradient is in FP32: 8 n eps
    tol = 18 * 2.0 ** -20 * np.abs(ref).max()
    assert np.abs(g[0]["D"].real - ref).max() <= tol
    maps = torch.tensor(eps[None], dtype=torch.float64, device="cuda", requires_grad=True)
    _, _, _, To, _ = autograd.solve_rt(maps, [(pw, {"D": ("pixmap", 0, 0.3), "U": ("uniform", 2.1, 0.7)}, same[2])],
                                       1.0 / f, np.zeros((2, 2)), which=np.zeros(2, int))
    To[:, 4].sum().backward()
    assert np.abs(maps.grad[0].cpu().numpy() - ref).max() <= tol
