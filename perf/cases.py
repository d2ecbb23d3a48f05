"""The work that users of this package have it do, as cases that can be timed and checked.

A case names a public entry point (``kind``) and its sizes; ``prepare`` makes the seeded inputs and
what a program keeps between calls, ``run`` makes one pass, ``exact`` restates the result in numpy /
torch complex128, and ``work`` counts the bytes and operations one pass cannot do without.
"""
import math

import numpy as np
import torch

from khepri_gb300 import autograd, batch
from khepri_gb300.crystal import Crystal
from khepri_gb300.twisted import TwistedBilayer

TWOPI = 2.0 * math.pi


def listed():
    return [
        # one frequency of the reference's own example: a disc slab at 5x5 harmonics through the
        # drop-in Crystal (set_source, solve, poynting_flux_end), the smallest call: pure latency
        dict(name="crystal_5x5", kind="crystal", stack="plain", px=5, py=5, lattice="square"),
        # the same loop body at a converged 11x11 basis on a five-layer stack
        dict(name="crystal_11x11", kind="crystal", stack="five", px=11, py=11, lattice="square"),
        # global S-matrix and per-order powers of a lossy slab on a hexagonal lattice: the complex128
        # layer S-matrices and star products that scattering and band-structure users read
        dict(name="smatrix_7x5_hex", kind="smatrix", stack="lossy", px=7, py=5, lattice="hexagonal"),
        # near fields of a slab on a substrate film on a 24 x 24 x 12 grid, after a solve
        dict(name="fields_5x5", kind="fields", stack="slab", px=5, py=5, lattice="square", grid=24, depths=12),
        # the reference's 151-frequency transmission spectrum in one batched call
        dict(name="sweep_5x5_151", kind="sweep", stack="plain", px=5, py=5, lattice="square", problems=151,
             chunk=256, method="mixed", both_pols=False),
        # oblique incidence on a lossy stack, both polarisations, rectangular basis
        dict(name="sweep_9x7_96", kind="sweep", stack="lossy", px=9, py=7, lattice="square", problems=96,
             chunk=256, method="mixed", both_pols=True),
        # the headline: frequency x Bloch-point sweep at 11x11, both polarisations, in calls of 912
        dict(name="sweep_11x11_1824", kind="sweep", stack="five", px=11, py=11, lattice="square", problems=1824,
             chunk=912, method="mixed", both_pols=True),
        # solve_rt's default method, the FP64 recursion
        dict(name="fp64_7x7_64", kind="sweep", stack="five", px=7, py=7, lattice="square", problems=64,
             chunk=256, method="gamma", both_pols=True),
        # diffraction efficiencies per order (the complex128 chain, batched)
        dict(name="orders_5x5_48", kind="orders", stack="lossy", px=5, py=5, lattice="square", problems=48),
        # many structures of uneven basis and layer count, one problem each (a dataset of devices)
        dict(name="uneven_32", kind="structures", count=32, max_px=13, max_layers=4),
        # one step of inverse design: R, T and the gradient of mean transmission for float32 maps
        dict(name="design_9x9_8x4", kind="design", px=9, py=9, designs=8, freqs=4),
        # a twisted bilayer at 3x3 base harmonics (81 in the product basis), both polarisations
        dict(name="twisted_3x3_8", kind="twisted", px=3, py=3, problems=8),
    ]


def _odd(rng, lo, hi):
    return rng.randrange(lo, hi + 1, 2)


def draw(rng):
    kind = rng.choice(["crystal", "smatrix", "fields", "sweep", "sweep", "sweep", "fp64", "orders", "structures",
                       "design", "twisted"])
    lat = rng.choice(["square", "square", "hexagonal"])
    if kind == "crystal":
        return dict(kind=kind, stack=rng.choice(["plain", "five", "lossy"]), px=_odd(rng, 1, 11), py=_odd(rng, 3, 11),
                    lattice=lat)
    if kind == "smatrix":
        return dict(kind=kind, stack=rng.choice(["plain", "five", "lossy"]), px=_odd(rng, 3, 9), py=_odd(rng, 3, 9),
                    lattice=lat)
    if kind == "fields":
        return dict(kind=kind, stack="slab", px=_odd(rng, 3, 5), py=_odd(rng, 3, 5),
                    lattice="square", grid=rng.randint(8, 40), depths=rng.randint(1, 16))
    if kind in ("sweep", "fp64", "orders"):
        most = {"sweep": 11, "fp64": 9, "orders": 7}[kind]
        px, py = _odd(rng, 3, most), _odd(rng, 3, most)
        hi = {"sweep": 912, "fp64": 96, "orders": 96}[kind]
        p = int(round(math.exp(rng.uniform(math.log(5), math.log(hi)))))
        c = dict(kind="orders" if kind == "orders" else "sweep", stack=rng.choice(["plain", "five", "lossy"]), px=px,
                 py=py, lattice=lat, problems=p)
        if kind != "orders":
            c.update(chunk=rng.choice([128, 256, 456]), method="mixed" if kind == "sweep" else "gamma",
                     both_pols=rng.random() < 0.5)
        return c
    if kind == "structures":
        return dict(kind=kind, count=rng.randint(6, 48), max_px=_odd(rng, 5, 13), max_layers=rng.randint(1, 6))
    if kind == "design":
        px = _odd(rng, 5, 9)
        return dict(kind=kind, px=px, py=px, designs=rng.randint(1, 12), freqs=rng.randint(1, 6))
    return dict(kind=kind, px=3, py=3, problems=rng.randint(2, 16))


# ------------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------------
def _blur(a, sigma):
    fx, fy = np.fft.fftfreq(a.shape[0])[:, None], np.fft.fftfreq(a.shape[1])[None, :]
    return np.fft.ifft2(np.fft.fft2(a) * np.exp(-2.0 * (math.pi * sigma) ** 2 * (fx * fx + fy * fy))).real


def _lossy_map(rng, n):
    return _blur(rng.uniform(1.0, 12.0, (n, n)), 4.0) - 1j * _blur(rng.uniform(0.0, 0.1, (n, n)), 4.0)


def _discs(rng, n):
    x = np.arange(n) / n
    X, Y = np.meshgrid(x, x, indexing="ij")
    inside = np.zeros((n, n), bool)
    for _ in range(int(rng.integers(1, 5))):
        dx, dy = X - rng.uniform(), Y - rng.uniform()
        dx, dy = dx - np.round(dx), dy - np.round(dy)
        inside |= dx * dx + dy * dy < rng.uniform(0.1, 0.3) ** 2
    return np.where(inside, 12.0, 1.0)


def _stack(name, rng):
    """layers, stack, epsi, epse of one device."""
    if name == "plain":  # [disc slab, spacer, disc slab]: the reference's plain crystal example
        x = np.linspace(-0.5, 0.5, 128)
        X, Y = np.meshgrid(x, x, indexing="ij")
        m = np.where(np.hypot(X, Y) < rng.uniform(0.3, 0.42), 1.0, 12.0)
        return ({"S1": ("uniform", 1.0, 1.1), "Scyl": ("pixmap", m, float(rng.uniform(0.4, 0.6)))},
                ["Scyl", "S1", "Scyl"], 1.0, 1.0)
    if name == "five":  # three slabs of one multi-disc map with two spacers, 256 x 256 pixels
        m, d, e = _discs(rng, 256), rng.uniform(0.2, 1.0, 5), rng.uniform(1.0, 4.0, 2)
        return ({"P1": ("pixmap", m, d[0]), "U1": ("uniform", e[0], d[1]), "P2": ("pixmap", m, d[2]),
                 "U2": ("uniform", e[1], d[3]), "P3": ("pixmap", m, d[4])}, ["P1", "U1", "P2", "U2", "P3"], 1.0, 1.0)
    if name == "slab":  # one disc slab on a film; thin, as the evanescent orders' fields grow with the depth
        x = np.linspace(-0.5, 0.5, 128)
        m = np.where(np.hypot(x[:, None], x[None, :]) < rng.uniform(0.2, 0.4), 1.0, 12.0)
        return ({"Film": ("uniform", 2.1, float(rng.uniform(0.1, 0.3))), "Slab": ("pixmap", m, float(rng.uniform(0.2, 0.4)))},
                ["Slab", "Film"], 1.0, 2.25)
    # two different lossy slabs on a substrate
    return ({"A": ("pixmap", _lossy_map(rng, 96), float(rng.uniform(0.2, 0.5))),
             "B": ("pixmap", _lossy_map(rng, 96), float(rng.uniform(0.2, 0.5))),
             "U": ("uniform", 2.1, float(rng.uniform(0.2, 0.5)))}, ["A", "U", "B"], 1.0, 2.25)


def _in_cone(rng, wl):
    """In-plane wave vectors inside 0.9 of the incidence light cone (R and T are defined there)."""
    k, a = 0.9 * TWOPI / wl * np.sqrt(rng.uniform(0, 1, wl.shape)), rng.uniform(0, TWOPI, wl.shape)
    return np.stack([k * np.cos(a), k * np.sin(a)], -1)


def _problems(c, rng, count):
    f = np.sort(rng.uniform(0.49, 0.60, count) if c.get("stack") == "plain" else rng.uniform(0.3, 0.7, count))
    wl = 1.0 / f
    return wl, np.zeros((count, 2)) if c.get("stack") == "plain" else _in_cone(rng, wl)


def _design(c, seed):
    rng = np.random.default_rng([seed, 5])
    theta = rng.standard_normal((c["designs"], 64, 64))
    f = np.sort(rng.uniform(0.4, 0.6, c["freqs"]))
    maps = (1.0 + 11.0 / (1.0 + np.exp(-theta))).astype(np.float32)
    which = np.repeat(np.arange(c["designs"]), c["freqs"])
    return maps, np.tile(1.0 / f, c["designs"]), which


def _uneven(c, seed):
    rng = np.random.default_rng([seed, 4])
    ents, wl = [], []
    for _ in range(c["count"]):
        p = int(rng.choice(np.arange(3, c["max_px"] + 1, 2)))
        nl = int(rng.integers(1, c["max_layers"] + 1))
        lay = {"L%d" % i: ("pixmap", _lossy_map(rng, 128), float(rng.uniform(0.2, 1.0))) for i in range(nl)}
        ents.append(((p, p), lay, list(lay)))
        wl.append(1.0 / rng.uniform(0.3, 0.8))
    wl = np.array(wl)
    return ents, wl, _in_cone(rng, wl)


def _twisted(c, seed):
    rng = np.random.default_rng([seed, 6])
    x = np.linspace(-0.5, 0.5, 64)
    X, Y = np.meshgrid(x, x, indexing="ij")
    m = np.where(np.hypot(X, Y) < rng.uniform(0.25, 0.4), 1.0, 4.0)
    wl = 1.0 / np.sort(rng.uniform(0.4, 0.8, c["problems"]))
    return ([("pixmap", m, 0.2)], [("uniform", 1.0, float(rng.uniform(0.1, 0.4)))], [("pixmap", m, 0.2)],
            math.radians(float(rng.uniform(5, 30))), wl, 0.3 * _in_cone(rng, wl))


def prepare(c, seed):
    kind = c["kind"]
    if kind == "structures":
        ents, wl, kp = _uneven(c, seed)
        return dict(c=c, ents=ents, wl=wl, kp=kp)
    if kind == "design":
        maps, wl, which = _design(c, seed)
        lay = lambda k: {"D1": ("pixmap", k, 0.3), "D2": ("pixmap", k, 0.3), "Sub": ("uniform", 2.1, 1.0)}  # noqa: E731
        ents = [((c["px"], c["py"]), lay(k), ["D1", "D2", "Sub"]) for k in range(c["designs"])]
        return dict(c=c, maps=torch.tensor(maps, device="cuda"), ents=ents, wl=wl, which=which)
    if kind == "twisted":
        lower, gap, upper, angle, wl, kp = _twisted(c, seed)
        return dict(c=c, tb=TwistedBilayer((c["px"], c["py"]), "square", angle, lower, gap, upper), wl=wl, kp=kp)
    rng = np.random.default_rng([seed, 1])
    layers, stack, epsi, epse = _stack(c["stack"], rng)
    wl, kp = _problems(c, rng, c.get("problems", 1))
    s = dict(c=c, layers=layers, stack=stack, epsi=epsi, epse=epse, wl=wl, kp=kp)
    if kind in ("crystal", "smatrix", "fields"):
        cl = Crystal((c["px"], c["py"]), lattice=c["lattice"], epsi=epsi, epse=epse)
        for name, (what, eps, d) in layers.items():
            (cl.add_layer_uniform if what == "uniform" else cl.add_layer_pixmap)(name, eps, d)
        cl.set_device(stack, kind == "fields")
        s["crystal"] = cl
    if kind == "fields":
        s["x"], s["y"], s["z"] = _grid(c, layers, stack)
    return s


def _grid(c, layers, stack):
    v = np.linspace(-0.5, 0.5, c["grid"])
    x, y = np.meshgrid(v, v, indexing="ij")
    total = sum(layers[n][2] for n in stack)
    return x, y, (np.arange(c["depths"]) + 0.5) / c["depths"] * total


def run(s):
    c = s["c"]
    kind = c["kind"]
    if kind in ("crystal", "smatrix", "fields"):
        cl = s["crystal"]
        cl.set_source(float(s["wl"][0]), 1.0, 0.5, kp=(s["kp"][0, 0], s["kp"][0, 1]))
        cl.solve()
        if kind == "crystal":
            return cl.poynting_flux_end()
        if kind == "smatrix":
            (r, ro), (t, to) = cl.poynting_flux_end(only_total=False)
            return r, t, ro, to, cl.S
        r, t = cl.poynting_flux_end()
        e, h = cl.fields_volume(s["x"], s["y"], s["z"])
        return r, t, e, h
    if kind == "sweep":
        return batch.solve_rt((c["px"], c["py"]), s["layers"], s["stack"], s["wl"], s["kp"], 1.0, 0.5,
                              lattice=c["lattice"], epsi=s["epsi"], epse=s["epse"], chunk=c["chunk"],
                              method=c["method"], both_pols=c["both_pols"])
    if kind == "orders":
        return batch.solve_rt((c["px"], c["py"]), s["layers"], s["stack"], s["wl"], s["kp"], 1.0, 0.5,
                              lattice=c["lattice"], epsi=s["epsi"], epse=s["epse"], orders=True)
    if kind == "structures":
        return batch.solve_structures(s["ents"], s["wl"], s["kp"], te=1.0, tm=0.5)
    if kind == "design":
        eps = s["maps"].detach().requires_grad_(True)
        r, t, ro, to, st = autograd.solve_rt(eps, s["ents"], s["wl"], np.zeros((len(s["wl"]), 2)), which=s["which"],
                                             te=1.0, tm=0.0)
        mid = (c["px"] * c["py"] - 1) // 2
        to[:, mid].mean().backward()
        return r.detach(), t.detach(), ro.detach(), to.detach(), eps.grad, st
    return s["tb"].solve_rt(s["wl"], s["kp"], both_pols=True)


# ------------------------------------------------------------------------------------------
# What a pass cannot do without.  One complex multiply-add is 8 operations: a patterned map's modes
# 117 n^3 per problem (eigenvectors 100, P Q 8, V 8, P 1), a patterned layer of the reflection
# recursion 53.3 n^3, a homogeneous one 10.7 n^3; a layer's S-matrix 85.3 n^3, a star product 82.7 n^3.
# ------------------------------------------------------------------------------------------
def _recursion(n, layers, stack):
    pat = [k for k in stack if layers[k][0] == "pixmap"]
    maps = len({id(layers[k][1]) for k in pat})
    return (117.0 * maps + 53.3 * len(pat) + 10.7 * (len(stack) - len(pat) + 1)) * n ** 3


def work(c):
    kind = c["kind"]
    if kind == "structures":
        ps = np.arange(3, c["max_px"] + 1, 2)
        mean = float(np.mean((2.0 * ps * ps) ** 3)) * (117.0 + 53.3) * (1 + c["max_layers"]) / 2
        maps = c["count"] * (1 + c["max_layers"]) / 2
        return dict(bytes=maps * 128 * 128 * 16 + c["count"] * 76, flops=c["count"] * mean)
    if kind == "twisted":
        n, N = 2 * c["px"] * c["py"], c["px"] * c["py"]
        per = N * 2 * (117.0 + 85.3 + 2 * 82.7) * n ** 3 + 8.0 / 3.0 * (n * N) ** 3
        return dict(bytes=2 * 64 * 64 * 8 + c["problems"] * 72, flops=c["problems"] * per)
    n = 2 * c["px"] * c["py"]
    if kind == "design":
        p = c["designs"] * c["freqs"]
        per = (117.0 + 2 * 53.3 + 2 * 10.7 + 20.0) * n ** 3
        return dict(bytes=2 * c["designs"] * 64 * 64 * 4 + p * (8 * n + 40), flops=p * per)
    layers, stack, _, _ = _stack(c["stack"], np.random.default_rng(0))
    pix = sum({id(v[1]): np.asarray(v[1]).nbytes for v in layers.values() if v[0] == "pixmap"}.values())
    p = c.get("problems", 1)
    pat = [k for k in stack if layers[k][0] == "pixmap"]
    chain = (117.0 * len({id(layers[k][1]) for k in pat}) + 85.3 * len({k for k in pat})
             + 82.7 * (len(stack) + 1)) * n ** 3
    if kind == "crystal":
        return dict(bytes=pix + 64, flops=_recursion(n, layers, stack))
    if kind == "smatrix":
        return dict(bytes=pix + 64 * n * n + 8 * n, flops=chain)
    if kind == "fields":
        pts = c["grid"] ** 2 * c["depths"] * 6
        return dict(bytes=pix + 16 * pts, flops=chain + 82.7 * (len(stack) + 1) * n ** 3 + 8.0 * pts * n / 2)
    if kind == "orders":
        return dict(bytes=pix + p * (56 + 8 * n + 20), flops=p * chain)
    return dict(bytes=pix + p * (72 + (36 if c["both_pols"] else 20)), flops=p * _recursion(n, layers, stack))


# ------------------------------------------------------------------------------------------
# The same results in 64 bits: dense RCWA with layer S-matrices and star products.  torch complex128
# throughout, so that autograd gives the design case's gradient.
# ------------------------------------------------------------------------------------------
def _diag(*d):
    a, b, c, e = (torch.diag(v) for v in d)
    return torch.cat([torch.cat([a, b], 1), torch.cat([c, e], 1)], 0)


def _lattice(name):
    h = math.sqrt(3) / 2
    a = np.eye(2) if name == "square" else np.array([[h, 0.5], [h, -0.5]])
    return TWOPI * np.linalg.inv(a).T


def _gvec(px, py, lattice):
    rec = _lattice(lattice)
    m, n = np.meshgrid(np.arange(px) - px // 2, np.arange(py) - py // 2)
    return rec[0][:, None] * m.ravel() + rec[1][:, None] * n.ravel()


def _conv(eps, px, py):
    eps = torch.as_tensor(eps).to(torch.complex128)
    f = torch.fft.fft2(eps) / eps.numel()
    r = np.arange(px * py)
    p, q = r % px, r // px
    return f[(p[:, None] - p[None]) % eps.shape[0], (q[:, None] - q[None]) % eps.shape[1]]


def _star(a, b):
    e = torch.eye(a[0].shape[0], dtype=torch.complex128)
    x = torch.linalg.solve(e - b[0] @ a[3], torch.cat([b[0] @ a[2], b[1]], 1))
    n = a[0].shape[0]
    u, v = x[:, :n], x[:, n:]
    y = torch.linalg.solve(e - a[3] @ b[0], torch.cat([a[2], a[3] @ b[1]], 1))
    return a[0] + a[1] @ u, a[1] @ v, b[2] @ y[:, :n], b[3] + b[2] @ y[:, n:]


def _kz(arg):
    return torch.where(arg.real < 0, -1j * torch.sqrt(-arg), torch.sqrt(arg))


def _device_s(kx, ky, k0, layers, epsi, epse):
    """S-matrices of [incidence, layers..., emergence] and their (W, V, lam); a layer is (C or eps, depth)."""
    nh, one = len(kx), torch.ones_like(kx)
    eye = torch.eye(2 * nh, dtype=torch.complex128)

    def homog(eps):
        return _diag(kx * ky, eps - kx ** 2, ky ** 2 - eps, -ky * kx)

    l0 = 1j * _kz(1 - kx ** 2 - ky ** 2).repeat(2)
    v0 = homog(one) / l0
    out = []
    for side, eps in (("inc", epsi), ("trn", epse)):
        lam = 1j * torch.conj(torch.sqrt(eps - kx ** 2 - ky ** 2)).repeat(2)
        v = homog(eps * one) / lam
        g = torch.linalg.solve(v0, v)
        a, b = eye + g, eye - g
        ai = torch.linalg.inv(a)
        s = (-ai @ b, 2 * ai, 0.5 * (a - b @ ai @ b), b @ ai)
        out.append((s if side == "inc" else (s[3], s[2], s[1], s[0]), eye, v, lam))
    mid, seen = [], {}
    for eps, depth in layers:
        if torch.is_tensor(eps):
            if id(eps) not in seen:
                ic = torch.linalg.inv(eps)
                ix, iy = ic * kx, ic * ky
                e, cx, cy = torch.eye(nh, dtype=torch.complex128), kx[:, None], ky[:, None]
                p = torch.cat([torch.cat([cx * iy, e - cx * ix], 1), torch.cat([cy * iy - e, -cy * ix], 1)], 0)
                q = torch.cat([torch.cat([torch.diag(kx * ky), eps - torch.diag(kx * kx)], 1),
                               torch.cat([torch.diag(ky * ky) - eps, -torch.diag(ky * kx)], 1)], 0)
                mu, w = torch.linalg.eig(p @ q)
                lam = torch.sqrt(mu)
                seen[id(eps)] = (w, (q @ w) / lam, lam)
            w, v, lam = seen[id(eps)]
        else:
            lam = 1j * _kz(eps - kx ** 2 - ky ** 2).repeat(2)
            w, v = eye, homog(eps * one) / lam
        t1, t2 = torch.linalg.inv(w), torch.linalg.solve(v, v0)
        a, b = t1 + t2, t1 - t2
        x = torch.exp(-lam * depth * k0)[:, None]
        aib = torch.linalg.solve(a, b)
        xb = x * b
        y = torch.linalg.solve(a, x * a)
        m = a - xb @ torch.linalg.solve(a, xb)
        s11, s12 = torch.linalg.solve(m, xb @ y - b), torch.linalg.solve(m, x * (a - b @ aib))
        mid.append(((s11, s12, s12, s11), w, v, lam))
    return [out[0]] + mid + [out[1]], v0


def _source(te, tm, kp, k0, epsi):
    kz = np.conj(np.sqrt(complex(k0 * k0 * epsi - kp[0] ** 2 - kp[1] ** 2)))
    k = np.array([kp[0], kp[1], kz]) / np.linalg.norm([kp[0], kp[1], kz])
    if np.linalg.norm(kp) < 1e-8:
        ate, atm = np.array([1, 0, 0], complex), np.array([0, 1, 0], complex)
    else:
        ate = np.array([-k[1], k[0], 0]) / np.linalg.norm([k[0], k[1]])
        atm = np.cross(ate, k)
        atm = atm / np.linalg.norm(atm)
    return (te * ate + tm * atm) / math.hypot(te, tm), kz


def _fluxes(s, col, kx, ky, kz_i, k0, eps):
    """Per-order powers of the outgoing amplitudes s @ col in a medium eps."""
    nh = len(kx)
    o = s @ col
    kz = torch.conj(torch.sqrt(eps - kx ** 2 - ky ** 2))
    sx, sy = o[:nh], o[nh:]
    sz = -(kx * sx + ky * sy) / kz
    return kz.real / float((kz_i / k0).real) * (sx.abs() ** 2 + sy.abs() ** 2 + sz.abs() ** 2)


def _solve(g, layers, wl, kp, pols, epsi, epse):
    """S, per-order R and T for every (te, tm) of pols."""
    k0 = TWOPI / wl
    kx = torch.as_tensor((kp[0] + g[0]) / k0).to(torch.complex128)
    ky = torch.as_tensor((kp[1] + g[1]) / k0).to(torch.complex128)
    parts, v0 = _device_s(kx, ky, k0, layers, epsi, epse)
    s = parts[0][0]
    for p in parts[1:]:
        s = _star(s, p[0])
    nh, got = len(kx), []
    for te, tm in pols:
        e, kz = _source(te, tm, kp, k0, epsi)
        col = torch.zeros(2 * nh, dtype=torch.complex128)
        col[(nh - 1) // 2], col[nh + (nh - 1) // 2] = e[0], e[1]
        got.append((_fluxes(s[0], col, kx, ky, kz, k0, epsi), _fluxes(s[2], col, kx, ky, kz, k0, epse)))
    return s, got, (parts, v0, kx, ky, k0, col)


def _as_layers(layers, stack, px, py):
    c = {}
    for name in stack:
        what, e, _ = layers[name]
        if what == "pixmap" and id(e) not in c:
            c[id(e)] = _conv(e, px, py)
    return [(c[id(layers[k][1])] if layers[k][0] == "pixmap" else layers[k][1], layers[k][2]) for k in stack]


def _exact_fields(c, st, layers, g):
    """E, H of the fields case: amplitudes from the chains on either side of each layer."""
    parts, v0, kx, ky, k0, col = st["tail"]
    s = [p[0] for p in parts]
    nh, n = len(kx), 2 * len(kx)
    eye, zero = torch.eye(n, dtype=torch.complex128), torch.zeros(n, n, dtype=torch.complex128)
    depth = [0.0] + [d for _, d in layers] + [0.0]
    start = np.concatenate([[0.0], np.cumsum(depth)[:-1]])
    x, y, zs = _grid(c, st["layers"], st["stack"])
    phase = torch.exp(1j * (k0 * (kx[:, None] * torch.as_tensor(x.ravel()) + ky[:, None] * torch.as_tensor(y.ravel()))))
    r0 = torch.cat([torch.cat([eye, eye], 1), torch.cat([-v0, v0], 1)], 0)
    rows = []
    for z in zs:
        i = int(np.searchsorted(start[1:], z))
        left = s[0]
        for p in s[1:i + 1]:
            left = _star(left, p)
        right = (zero, eye, eye, zero)
        for p in reversed(s[i + 1:]):
            right = _star(p, right)
        cp = torch.linalg.solve(eye - left[3] @ right[0], left[2] @ (0.5 * col))
        _, w, v, lam = parts[i]
        ri = torch.cat([torch.cat([w, w], 1), torch.cat([-v, v], 1)], 0)
        zb = k0 * (depth[i] - (z - start[i]))
        prop = torch.cat([torch.exp(lam * zb), torch.exp(-lam * zb)])
        f = ri @ (prop * torch.linalg.solve(ri, r0 @ torch.cat([cp, right[0] @ cp])))
        sx, sy, ux, uy = f[:nh], f[nh:n], f[n:n + nh], f[n + nh:]
        rhs, eps = kx * uy - ky * ux, layers[i - 1][0]
        sz = -1j * (torch.linalg.solve(eps, rhs) if torch.is_tensor(eps) else rhs / eps)
        uz = -1j * (kx * sy - ky * sx)
        rows.append(torch.stack([q @ phase for q in (sx, sy, sz, ux, uy, uz)]))
    f = torch.stack(rows).reshape(len(zs), 6, *x.shape).numpy()
    return f[:, :3], f[:, 3:]


def _cost(c):
    """Rough seconds that ``exact`` takes."""
    if c["kind"] == "structures":
        return c["count"] * (1 + c["max_layers"]) / 2 * 2e-8 * np.mean((2.0 * np.arange(3, c["max_px"] + 1, 2) ** 2) ** 3)
    if c["kind"] == "twisted":
        return c["problems"] * 0.3
    p = c.get("problems", 1) if c["kind"] != "design" else 2 * c["designs"] * c["freqs"]
    return p * (0.01 + 3e-8 * (2.0 * c["px"] * c["py"]) ** 3)


def exact(c, seed):
    if _cost(c) > 20:
        return None
    kind = c["kind"]
    if kind == "structures":
        ents, wl, kp = _uneven(c, seed)
        r = []
        for (pw, lay, st), w, k in zip(ents, wl, kp):
            _, got, _ = _solve(_gvec(*pw, "square"), _as_layers(lay, st, *pw), w, k, [(1.0, 0.5)], 1.0, 1.0)
            r.append([float(v.sum()) for v in got[0]])
        r = np.array(r)
        return r[:, 0], r[:, 1], None
    if kind == "design":
        maps, wl, which = _design(c, seed)
        eps = torch.tensor(maps, dtype=torch.float64, requires_grad=True)
        g = _gvec(c["px"], c["py"], "square")
        conv = [_conv(e, c["px"], c["py"]) for e in eps]
        ro, to = [], []
        for w, k in zip(wl, which):
            _, got, _ = _solve(g, [(conv[k], 0.3), (conv[k], 0.3), (2.1, 1.0)], w, (0.0, 0.0), [(1.0, 0.0)], 1.0, 1.0)
            ro.append(got[0][0])
            to.append(got[0][1])
        ro, to = torch.stack(ro), torch.stack(to)
        to[:, (c["px"] * c["py"] - 1) // 2].mean().backward()
        ro, to = ro.detach(), to.detach()
        return ro.sum(1), to.sum(1), ro, to, eps.grad, None
    if kind == "twisted":
        lower, gap, upper, angle, wl, kp = _twisted(c, seed)
        g1 = _gvec(c["px"], c["py"], "square")
        ca, sa = math.cos(angle), math.sin(angle)
        g2 = np.array([[ca, -sa], [sa, ca]]) @ g1
        g = (g1[:, :, None] + g2[:, None, :]).reshape(2, -1)
        m = _conv(lower[0][1], c["px"], c["py"])
        e = torch.eye(m.shape[0], dtype=torch.complex128)
        lay = [(torch.kron(m, e), lower[0][2]), (gap[0][1], gap[0][2]), (torch.kron(e, m), upper[0][2])]
        both = np.array([[[float(v.sum()) for v in p] for p in _solve(g, lay, w, k, [(1.0, 0.0), (0.0, 1.0)], 1.0, 1.0)[1]]
                         for w, k in zip(wl, kp)])
        return both[:, :, 0], both[:, :, 1], None
    rng = np.random.default_rng([seed, 1])
    layers, stack, epsi, epse = _stack(c["stack"], rng)
    wl, kp = _problems(c, rng, c.get("problems", 1))
    g = _gvec(c["px"], c["py"], c["lattice"])
    lay = _as_layers(layers, stack, c["px"], c["py"])
    pols = [(1.0, 0.0), (0.0, 1.0)] if c.get("both_pols") else [(1.0, 0.5)]
    all_rt, all_o = [], []
    for w, k in zip(wl, kp):
        s, got, tail = _solve(g, lay, w, k, pols, epsi, epse)
        all_rt.append([[float(v.sum()) for v in p] for p in got])
        all_o.append([v.numpy() for v in got[0]])
    rt = np.array(all_rt)  # [P, npol, 2]
    if kind == "crystal":
        return float(rt[0, 0, 0]), float(rt[0, 0, 1])
    if kind == "smatrix":
        full = torch.stack([torch.stack([s[0], s[1]]), torch.stack([s[2], s[3]])])
        return float(rt[0, 0, 0]), float(rt[0, 0, 1]), all_o[0][0], all_o[0][1], full
    if kind == "fields":
        e, h = _exact_fields(c, dict(tail=tail, layers=layers, stack=stack), lay, g)
        return float(rt[0, 0, 0]), float(rt[0, 0, 1]), e, h
    if kind == "orders":
        o = np.array(all_o)
        return rt[:, 0, 0], rt[:, 0, 1], o[:, 0], o[:, 1], None
    if c["both_pols"]:
        return rt[:, :, 0], rt[:, :, 1], None
    return rt[:, 0, 0], rt[:, 0, 1], None
