"""The eigensolver's QR sweep in windows of 31 rotations (32 columns): sizes whose first sweeps end just
below, at and just above one, two and three windows, several problems per call so that no CTA starts
from another's shared memory alone.  No problem may need a re-solve, and R and T match the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pw", [(1, 1), (1, 15), (1, 17), (5, 5), (1, 31), (3, 11), (1, 47), (7, 7), (9, 7), (13, 13)])
def test_no_problem_needs_a_resolve(pw):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import __graft_entry__
    __graft_entry__.build()
    from khepri_gb300 import batch, workloads
    from oracle import khepri_oracle as ko
    rng = np.random.default_rng(sum(pw))
    m = workloads.periodic_gaussian_blur(rng.uniform(1, 12, (128, 128)), 4.0) - 0.02j
    layers = {"A": ("pixmap", m, 0.3), "U": ("uniform", 2.0, 0.2)}
    P = 200 if pw[0] * pw[1] < 60 else 12
    f = rng.uniform(0.35, 0.65, P)
    a, k = rng.uniform(0, 2 * np.pi, P), 0.8 * 2 * np.pi * f * np.sqrt(rng.uniform(0, 1, P))
    kp = np.stack([k * np.cos(a), k * np.sin(a)], 1)
    before = dict(batch.STATS)
    R, T, st = batch.solve_rt(pw, layers, ["A", "U"], 1.0 / f, kp, 1.0, 0.5, method="mixed")
    assert not st.any() and batch.STATS == before
    for i in range(2):
        r, t = ko.solve_rt(pw, layers, ["A", "U"], 1.0 / f[i], 1.0, 0.5, kp=kp[i])
        assert abs(R[i] - r) < 1e-8 and abs(T[i] - t) < 1e-8  # the modes' residual test accepts 1e-8
