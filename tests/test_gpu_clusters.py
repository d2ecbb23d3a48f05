"""Eigenvalue clusters of the mixed path's refinement: nearly uniform symmetric maps at normal
incidence, whose modes fall into exactly degenerate pairs and into groups of close eigenvalues below,
at and above the largest cluster taken as one block, against the CPU oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pw", [(1, 1), (1, 3), (3, 3), (5, 5), (7, 5)])
@pytest.mark.parametrize("contrast", [1e-6, 1e-3, 0.3])
def test_close_eigenvalues_match_the_oracle(pw, contrast):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import __graft_entry__
    __graft_entry__.build()
    from khepri_gb300 import batch, workloads
    from oracle import khepri_oracle as ko
    m = workloads.disc_canvas(48, 0.3, 2.0 + contrast, 2.0)
    layers = {"A": ("pixmap", m, 0.4), "U": ("uniform", 1.5, 0.3)}
    wl = 1.0 / np.array([0.41, 0.57])
    kp = np.zeros((2, 2))
    R, T, st = batch.solve_rt(pw, layers, ["A", "U"], wl, kp, 1.0, 0.5, method="mixed")
    assert not st.any()
    for i, w in enumerate(wl):
        r, t = ko.solve_rt(pw, layers, ["A", "U"], w, 1.0, 0.5, kp=(0.0, 0.0))
        # the modes' residual test accepts 1e-8; R and T are bounded functions of the modes
        assert abs(R[i] - r) < 1e-8 and abs(T[i] - t) < 1e-8
