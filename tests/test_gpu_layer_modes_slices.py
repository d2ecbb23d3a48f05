"""FP64 modes of calls whose matrices the eigensolver takes a part at a time (its scratch stays within a
bound), ordinary maps beside nearly uniform ones, which the FP64 eigensolver solves for the whole call
afterwards: eigenpair residuals in torch, FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pw,batch", [((3, 3), 7), ((11, 11), 200)])
def test_modes_are_eigenpairs(pw, batch):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import __graft_entry__
    __graft_entry__.build()
    from khepri_gb300 import _capi, engine, workloads
    lib = _capi.load()
    st = engine.StructureGPU(pw, engine.lattice_vectors("square"))
    nh, n = st.nh, st.n
    maps = [st.prepare_map(workloads.disc_canvas(64, 0.35, 1.0, e)) for e in (12.0, 1.000001)]
    conv, hx, hy = (torch.cat([m[k].reshape(1, nh, nh) for m in maps]).contiguous() for k in ("conv", "hx", "hy"))
    near = np.zeros(batch, dtype=np.int32)
    near[[1, batch // 2, batch - 1]] = 1
    mi = torch.from_numpy(near).cuda()
    wl = 1.0 / np.linspace(0.37, 0.61, batch)
    prob = engine.Problems.make(wl, np.zeros((batch, 2)), 1.0, 0.0, "cuda")
    W = torch.full((batch, n, n), float("nan"), dtype=torch.complex128, device="cuda")
    V, lam = torch.empty_like(W), torch.empty((batch, n), dtype=torch.complex128, device="cuda")
    status = torch.zeros(batch, dtype=torch.int32, device="cuda")
    ws = torch.empty(lib.khp_layer_modes_workspace(batch, nh), dtype=torch.uint8, device="cuda")
    _capi.check(lib.khp_layer_modes(batch, nh, _capi.ptr(mi), _capi.ptr(conv), _capi.ptr(hx), _capi.ptr(hy),
                                    _capi.ptr(st.gx), _capi.ptr(st.gy), _capi.ptr(prob.kp), _capi.ptr(prob.k0),
                                    _capi.ptr(W), _capi.ptr(V), _capi.ptr(lam), _capi.ptr(status), _capi.ptr(ws),
                                    ws.numel(), _capi.stream_ptr()), "khp_layer_modes")
    assert not status.any()
    eye = torch.eye(nh, dtype=torch.complex128, device="cuda")
    gx, gy = st.gx.to(torch.complex128), st.gy.to(torch.complex128)
    ics = [torch.linalg.inv(c) for c in conv]
    worst = 0.0
    for b in range(batch):
        C, ic, k0 = conv[near[b]], ics[near[b]], 2 * np.pi / wl[b]
        x, y = gx / k0, gy / k0
        X, Y = x[:, None], y[:, None]
        P = torch.cat([torch.cat([X * ic * y, eye - X * ic * x], 1), torch.cat([Y * ic * y - eye, -Y * ic * x], 1)])
        Q = torch.cat([torch.cat([torch.diag(x * y), C - torch.diag(x * x)], 1),
                       torch.cat([torch.diag(y * y) - C, -torch.diag(x * y)], 1)])
        mu = lam[b] ** 2
        r = (P @ (Q @ W[b]) - W[b] * mu).abs().amax(0) / (mu.abs().max() * W[b].abs().amax(0))
        worst = max(worst, float(r.max()))
    # twice and a half what the solver accepts, 4e-16 n (its own and this test's rounding of P Q W)
    assert worst <= 1e-15 * n, worst
