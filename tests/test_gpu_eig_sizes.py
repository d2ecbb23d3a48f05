"""The FP32 eigensolver at the sizes and batches where its forms change: Hessenberg clusters of 16 CTAs, one
CTA per matrix for hundreds of matrices whose cluster CTAs would fill their SMs and beyond what a cluster
holds, strips of the QR in more than one pass, eigenvectors in the QR's CTA, and the QR teams for more than
two matrices per SM.  No problem may need a re-solve (an FP32 failure would), R and T match the oracle or
conserve energy; the FP32 inverses at the panel widths between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def built():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import __graft_entry__
    __graft_entry__.build()


@pytest.mark.parametrize("pw,problems,check", [
    ((15, 17), 2, 1),    # n = 510: a cluster of 16
    ((17, 17), 3, 1),    # n = 578: the same
    ((17, 19), 2, 1),    # n = 646: no cluster, two passes of strips
    ((17, 25), 1, 0),    # n = 850: eigenvectors in the QR's CTA
    ((13, 11), 260, 1),  # n = 286: more than 256 matrices of whole-SM cluster CTAs
    ((9, 9), 310, 1),    # n = 162: QR teams of 288
    ((7, 7), 310, 1),    # n = 98: QR teams of 192
])
def test_no_problem_needs_a_resolve(built, pw, problems, check):
    from khepri_gb300 import batch, workloads
    from oracle import khepri_oracle as ko
    rng = np.random.default_rng(sum(pw))
    m = workloads.periodic_gaussian_blur(rng.uniform(1, 12, (128, 128)), 4.0)
    layers = {"A": ("pixmap", m, 0.3), "U": ("uniform", 2.0, 0.2)}
    f = rng.uniform(0.35, 0.65, problems)
    a, k = rng.uniform(0, 2 * np.pi, problems), 0.8 * 2 * np.pi * f * np.sqrt(rng.uniform(0, 1, problems))
    kp = np.stack([k * np.cos(a), k * np.sin(a)], 1)
    before = dict(batch.STATS)
    R, T, st = batch.solve_rt(pw, layers, ["A", "U"], 1.0 / f, kp, 1.0, 0.5, method="mixed", chunk=problems)
    assert not st.any() and batch.STATS == before
    assert np.abs(R + T - 1).max() < 1e-7  # lossless; the modes' residual test accepts 1e-8
    for i in range(check):
        r, t = ko.solve_rt(pw, layers, ["A", "U"], 1.0 / f[i], 1.0, 0.5, kp=kp[i])
        assert abs(R[i] - r) < 1e-8 and abs(T[i] - t) < 1e-8


@pytest.mark.parametrize("n", [720, 800, 900, 1000])
def test_fp32_inverse_panel_widths(built, n):
    import torch
    from khepri_gb300 import _capi
    lib = _capi.load()
    rng = np.random.default_rng(n)
    A = rng.standard_normal((2, n, n)) + 1j * rng.standard_normal((2, n, n)) + 0.5 * np.sqrt(n) * np.eye(n)
    a = torch.from_numpy(A).to(torch.complex64).cuda()
    ref = torch.linalg.inv(a.to(torch.complex128))
    cond = torch.linalg.cond(a.to(torch.complex128))
    x, st = torch.empty_like(a), torch.zeros(2, dtype=torch.int32, device="cuda")
    ws = torch.empty(lib.khp_inverse_workspace(2, n), dtype=torch.uint8, device="cuda")
    _capi.check(lib.khp_inverse_gj(2, n, 1, _capi.ptr(a), n * n, _capi.ptr(x), n * n, _capi.ptr(st), _capi.ptr(ws),
                                   ws.numel(), _capi.stream_ptr()), "khp_inverse_gj")
    assert not st.any()
    err = (x.to(torch.complex128) - ref).abs().amax((1, 2)) / ref.abs().amax((1, 2))
    assert (err <= 8 * n * 2.0 ** -23 * cond).all(), (err, cond)  # c n eps cond
