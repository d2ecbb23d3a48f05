"""FP64 modes of a patterned layer (khp_layer_modes) by the refined FP32 eigensolver: residual of P Q
computed in numpy, at the sizes around the change from the FP64 eigensolver, for ordinary maps and for
nearly uniform symmetric ones, whose degenerate groups fail the residual test and take the FP64
eigensolver; unit columns either way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pw", [(1, 1), (1, 5), (7, 1), (3, 3), (5, 3), (7, 7)])
@pytest.mark.parametrize("kind", ["disc", "lossy", "near"])
def test_modes_are_eigenpairs(pw, kind):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import __graft_entry__
    __graft_entry__.build()
    from khepri_gb300 import engine, workloads
    rng = np.random.default_rng(5)
    if kind == "lossy":
        m = workloads.periodic_gaussian_blur(rng.uniform(1, 12, (48, 48)), 3.0) - 0.1j
    else:
        m = workloads.disc_canvas(48, 0.35, 1.0, 12.0 if kind == "disc" else 1.000001)
    wl = 1.0 / np.array([0.37, 0.52, 0.61])
    kp = np.zeros((3, 2)) if kind != "lossy" else np.array([[0.5, 0.2], [-1.0, 0.3], [0.1, 1.9]])
    st = engine.StructureGPU(pw, engine.lattice_vectors("square"))
    prob = engine.Problems.make(wl, kp, 1.0, 0.0, "cuda")
    status = torch.zeros(3, dtype=torch.int32, device="cuda")
    entry = st.prepare_map(m)
    W, _, lam = (t.cpu().numpy() for t in engine.layer_modes(st, entry, prob, status))
    assert not status.any()
    C = entry["conv"][0].cpu().numpy()
    n = 2 * C.shape[0]
    gx, gy = st.gx.cpu().numpy(), st.gy.cpu().numpy()
    eye, ic = np.eye(n // 2), np.linalg.inv(C)
    for b in range(3):
        k0 = 2 * np.pi / wl[b]
        x, y = (kp[b, 0] + gx) / k0, (kp[b, 1] + gy) / k0
        P = np.block([[x[:, None] * ic * y, eye - x[:, None] * ic * x], [y[:, None] * ic * y - eye, -y[:, None] * ic * x]])
        Q = np.block([[np.diag(x * y), C - np.diag(x * x)], [np.diag(y * y) - C, -np.diag(x * y)]])
        mu = lam[b] ** 2
        r = np.abs(P @ (Q @ W[b]) - W[b] * mu).max(axis=0) / (np.abs(mu).max() * np.abs(W[b]).max(axis=0))
        # backward error of an FP64 eigensolver, c n eps
        assert r.max() <= 50 * n * 2.0 ** -52, (pw, kind, r.max())
        assert np.abs(np.linalg.norm(W[b], axis=0) - 1).max() < 1e-13
