"""Gradient of the problem that the gradient call solves again with more rounds (the design of
test_gpu_grad_repair.py at f = 0.48 c/a, where a round of the stack's refinement gains a factor of a few),
against torch autograd through the complex128 restatement of the reference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_repaired_gradient_matches_autograd(khp):
    import torch
    from khepri_gb300 import batch, workloads
    from oracle import torch_c128
    _, structs, freqs = workloads.inverse_design(44, seed=0)
    s, f = structs[43], float(freqs[6])
    eps = torch.tensor(s.layers["D1"][1], dtype=torch.float64, requires_grad=True)
    layers = {"D1": ("pixmap", eps, 0.3), "D2": ("pixmap", eps, 0.3), "Sub": ("uniform", 2.1, 1.0)}
    _, _, _, t_orders = torch_c128.solve_orders(s.pw, layers, s.stack, 1.0 / f)
    t_orders[40].backward()
    ref, t_ref = eps.grad.numpy(), float(t_orders[40].detach())
    dT = np.zeros((1, 81))
    dT[0, 40] = 1.0
    before = batch.STATS["grad_repairs"]
    _, _, _, To, grads, st = batch.solve_structures_grad([(s.pw, s.layers, s.stack)], np.array([1.0 / f]),
                                                         np.zeros((1, 2)), which=np.zeros(1, int), dT=dT)
    assert batch.STATS["grad_repairs"] == before + 1 and not st.any()
    assert abs(To[0, 40] - t_ref) < 1e-8  # the refinement accepts 1e-9
    # the contraction W H^T W^-1 of the gradient is in FP32: n roundings of an entry
    assert np.abs(grads[0]["D1"].real - ref).max() <= 162 * 2.0 ** -23 * np.abs(ref).max()
