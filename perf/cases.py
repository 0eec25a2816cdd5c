"""Performance cases of the framework: the far-field sum and the RCWA solves as a
metalens design program calls them, over the sizes it meets.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program holds before the call (inputs on the GPU, or
                        host arrays for the host-buffer calls, and cell descriptors)
    run(state)          one pass through the public entry points
    work(case)          bytes and flops no implementation can do without
    exact(case, seed)   what run returns, in plain FP64 torch / numpy

Far-field inputs are metalens apertures (lattice sites in a disc, hyperbolic
phase, |t| ~ U[0.85, 1]); RCWA inputs are pillars in a square or rectangular
period with seeded fills, heights and indices.
"""
import math

import numpy as np
import torch

from celeris_b200 import capi, torch_ops, workloads

FORMS = {"plain": capi.FORM_PLAIN_F64, "precision": capi.FORM_F32C}
SHAPES = (capi.SHAPE_RECT, capi.SHAPE_ELLIPSE, capi.SHAPE_RING)


def listed():
    return [
        # a small lens looked at once from host arrays: the call's latency
        dict(name="psf_small", kind="psf_host", lattice=37, n=41),
        # the 70,688-pillar lens on its 161^2 focal grid, device arrays, both forms
        dict(name="psf_plain", kind="psf", form="plain", lattice=300, n=161),
        dict(name="psf_precision", kind="psf", form="precision", lattice=300, n=161),
        # the largest single-GPU far field: 785,456 pillars on 1024^2 pixels
        dict(name="psf_large", kind="psf", form="precision", lattice=1000, n=1024),
        # through-focus analysis: the x-z caustic of the 70k lens on 201 x 201 points
        dict(name="caustic", kind="zx", lattice=300, nx=201, nz=201),
        # inverse design: fills -> t by splines, field, encircled energy, adjoint
        dict(name="design_plain", kind="design", form="plain", lattice=300, n=161),
        dict(name="design_precision", kind="design", form="precision", lattice=300, n=161),
        # one unit cell, as a trial solve or a step of a height search makes it
        dict(name="cell", kind="cell", M=5),
        # the 64-width library sweep
        dict(name="library", kind="library", ncell=64, M=3),
        # a freeform library: rasterised squares, circles and rings, M = 3..7
        dict(name="uneven", kind="uneven", ncell=512, M=3, M_max=7, grid=256),
        # angular response of a library: oblique incidence, no mirror symmetry
        dict(name="oblique", kind="oblique", ncell=96, M=4),
        # pillars on a patterned second layer
        dict(name="stack", kind="stack", ncell=64, layers=2, M=3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["psf_host", "psf", "psf", "zx", "design", "cell", "library", "uneven", "oblique", "stack"])
    if kind == "psf_host":
        return dict(kind=kind, lattice=_log_int(rng, 9, 300), n=_log_int(rng, 11, 161))
    if kind == "psf":
        form = rng.choice(sorted(FORMS))
        return dict(kind=kind, form=form, lattice=_log_int(rng, 30, 600), n=_log_int(rng, 31, 321))
    if kind == "zx":
        return dict(kind=kind, lattice=_log_int(rng, 30, 300), nx=_log_int(rng, 21, 301), nz=_log_int(rng, 21, 301))
    if kind == "design":
        form = rng.choice(sorted(FORMS))
        return dict(kind=kind, form=form, lattice=_log_int(rng, 60, 400), n=_log_int(rng, 41, 201))
    if kind == "cell":
        return dict(kind=kind, M=rng.randint(1, 7))
    if kind == "library":
        return dict(kind=kind, ncell=_log_int(rng, 8, 400), M=rng.randint(2, 6))
    if kind == "uneven":
        return dict(kind=kind, ncell=_log_int(rng, 24, 512), M=rng.randint(2, 4), M_max=rng.randint(5, 7),
                    grid=rng.choice([0, 128, 256]))
    if kind == "oblique":
        return dict(kind=kind, ncell=_log_int(rng, 4, 160), M=rng.randint(2, 5))
    return dict(kind=kind, ncell=_log_int(rng, 4, 96), layers=rng.randint(2, 3), M=rng.randint(2, 4))


# ---- inputs ----------------------------------------------------------------------
def _aperture(case, seed):
    """A lens of lattice x lattice sites in a disc; the two sizes of the
    configurations (300 at 0.4 um, 1000 at 0.35 um) keep their own geometry, other
    sizes keep the smaller one's period and f-number."""
    n = case["lattice"]
    if n == 1000:
        return workloads.metalens_aperture(1000, 0.35, 175.0, 0.532, 1000.0, seed), 20.0
    radius = 0.2 * n
    return workloads.metalens_aperture(n, 0.4, radius, 0.633, radius / 0.6, seed), 5.0


def _spline_tables():
    """A 64-entry unit-cell library: transmission amplitude and phase over the fill."""
    fill = np.linspace(0.2, 0.9, 64)
    amp = 0.92 + 0.06 * np.cos(11.0 * fill)
    phase = 2.0 * np.pi * (fill - 0.2) / 0.7 + 0.3 * np.sin(5.0 * fill)
    return fill, amp, phase


def _fills(case, seed, npil):
    fill, _, _ = _spline_tables()
    return np.random.default_rng(seed + 7).uniform(fill[1], fill[-2], npil)


def _cells(case, seed):
    """Keyword sets of the case's cells (one per cell; per layer for stacks)."""
    rng = np.random.default_rng(seed)
    kind, M = case["kind"], case["M"]
    base = dict(period_um=0.4, wavelength_um=0.633, n_inc=1.0, n_sub=1.46, eps_pillar=4.0, eps_bg=1.0)
    if kind == "cell":
        return [dict(base, fill_x=float(rng.uniform(0.2, 0.9)), thickness_um=float(rng.uniform(0.4, 0.8)), Mx=M)]
    if kind == "library":
        h = float(rng.uniform(0.5, 0.7))
        return [dict(base, fill_x=float(f), thickness_um=h, Mx=M) for f in np.linspace(0.2, 0.9, case["ncell"])]
    if kind == "uneven":
        out = []
        for i in range(case["ncell"]):
            out.append(dict(base, wavelength_um=float(rng.uniform(0.45, 0.70)), eps_pillar=float(rng.uniform(1.9, 2.6)) ** 2,
                            fill_x=float(rng.uniform(0.15, 0.85)), thickness_um=float(rng.uniform(0.4, 0.9)),
                            Mx=M + i % (case["M_max"] + 1 - M), shape=SHAPES[int(rng.integers(0, 3))],
                            shape_param=0.5, grid=case["grid"], force_laurent=1))
        return out
    if kind == "oblique":
        h = float(rng.uniform(0.5, 0.7))
        return [dict(base, period_y_um=0.38, period_x_um=0.4, theta_rad=float(rng.uniform(0.05, 0.5)),
                     phi_rad=float(rng.uniform(0.0, 1.5)), fill_x=float(rng.uniform(0.25, 0.85)),
                     fill_y=float(rng.uniform(0.25, 0.85)), thickness_um=h, Mx=M) for _ in range(case["ncell"])]
    out = []
    for _ in range(case["ncell"]):
        wl = float(rng.uniform(0.5, 0.7))
        for layer in range(case["layers"]):
            out.append(dict(base, wavelength_um=wl, fill_x=float(rng.uniform(0.3, 0.85)),
                            fill_y=float(rng.uniform(0.3, 0.85)), thickness_um=float(rng.uniform(0.15, 0.6)), Mx=M,
                            eps_pillar=4.0 if layer % 2 == 0 else 2.25))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("psf_host", "psf", "zx", "design"):
        ap, half = _aperture(case, seed)
        state = dict(kind=kind, ap=ap, half=half, case=case)
        if kind in ("psf", "design"):
            state["px"] = torch.tensor(ap.px, device="cuda")
            state["py"] = torch.tensor(ap.py, device="cuda")
            state["grid"] = torch_ops.FarFieldGrid(case["n"], half, ap.focal_um, ap.wavelength_um)
            state["form"] = FORMS[case["form"]]
        if kind == "psf":
            state["t"] = torch.tensor(ap.t, device="cuda")
        if kind == "design":
            state["spline"] = torch_ops.LibrarySpline(*_spline_tables())
            state["w"] = torch.tensor(_fills(case, seed, ap.npil), device="cuda", requires_grad=True)
        return state
    cells = [capi.rcwa_cell(**c) for c in _cells(case, seed)]
    if kind == "stack":
        nl = case["layers"]
        cells = [cells[i:i + nl] for i in range(0, len(cells), nl)]
    return dict(kind=kind, cells=cells)


# ---- one pass ----------------------------------------------------------------------
def _table(results):
    """Per result (R, T, sum_de, de_t0, de_r0, tx0, ty0) as one complex row."""
    return np.array([tuple(r.values()) for r in results], dtype=np.complex128)


def run(state):
    kind = state["kind"]
    if kind == "psf_host":
        ap, n = state["ap"], state["case"]["n"]
        return capi.propagate_psf(ap.px, ap.py, ap.t, 0.0, 0.0, ap.focal_um, ap.k, n, state["half"])
    if kind == "psf":
        return torch_ops.rs_field_dev(state["px"], state["py"], state["t"], state["grid"], state["form"],
                                      want_intensity=True)
    if kind == "zx":
        ap, c, f = state["ap"], state["case"], state["ap"].focal_um
        return capi.propagate_zx(ap.px, ap.py, ap.t, -state["half"], state["half"], c["nx"], 0.8 * f, 1.2 * f,
                                 c["nz"], ap.k)
    if kind == "design":
        w = state["w"]
        w.grad = None
        E = torch_ops.rs_field(state["spline"](w), state["px"], state["py"], state["grid"], state["form"])
        loss = torch_ops.encircled_energy_loss(E, state["grid"], 1.0)
        loss.backward()
        return E.detach(), loss.detach(), w.grad
    if kind == "cell":
        return _table([capi.solve_rcwa_2d(state["cells"][0])])
    if kind == "stack":
        results, info = capi.rcwa_stack_batch(state["cells"])
    else:
        results, info = capi.rcwa_batch(state["cells"])
    return _table(results), info


# ---- what one pass cannot do without ---------------------------------------------------
def _class_order(M):
    return (M + 1) ** 2 + M ** 2


def work(case):
    kind = case["kind"]
    if kind in ("psf_host", "psf", "zx", "design"):
        npil = float(workloads.metalens_aperture(case["lattice"], 1.0, 0.5 * case["lattice"], 1.0, 1.0).npil)
        npix = float(case["nx"] * case["nz"] if kind == "zx" else case["n"] ** 2)
        out = {"psf_host": 8, "zx": 8, "psf": 24, "design": 16}[kind]
        passes = 2 if kind == "design" else 1  # forward and adjoint
        # a term: distance 6, square root 1, phase 1, sine and cosine 2, division 1, complex product and sum 10
        return {"bytes": 32.0 * npil + out * npix + (16.0 * npil if kind == "design" else 0.0),
                "flops": 21.0 * npil * npix * passes}
    cells = 1 if kind == "cell" else case["ncell"] * case.get("layers", 1)
    orders = range(case["M"], case.get("M_max", case["M"]) + 1)
    # about 240 n^3 flops per eigenproblem and its interfaces; a cell with both
    # mirrors and the 90-degree rotation needs one class of a quarter of the order
    size = (lambda M: _class_order(M)) if kind in ("cell", "library", "uneven") else (lambda M: 2 * (2 * M + 1) ** 2)
    per = sum(240.0 * size(M) ** 3 for M in orders) / len(orders)
    return {"bytes": cells * 300.0, "flops": cells * per}


# ---- the same in plain 64-bit torch and numpy --------------------------------------------
def _blocks(npil, npix):
    step = max(1, (1 << 25) // max(1, npil))
    return [(a, min(npix, a + step)) for a in range(0, npix, step)]


def _field64(px, py, t, fx, fy, z, k):
    """E(p) = sum_j t_j e^{ikR} / R over flat pixel coordinates."""
    E = torch.empty(fx.numel(), dtype=torch.complex128, device=px.device)
    for a, b in _blocks(px.numel(), fx.numel()):
        dx, dy = fx[a:b, None] - px[None, :], fy[a:b, None] - py[None, :]
        R = torch.sqrt(dx * dx + dy * dy + (z[a:b, None] if z.numel() > 1 else z) ** 2)
        u, ph = 1.0 / R, k * R
        c, s = u * torch.cos(ph), u * torch.sin(ph)
        E[a:b] = torch.complex(c @ t.real - s @ t.imag, s @ t.real + c @ t.imag)
    return E


def _adjoint64(px, py, v, fx, fy, z, k):
    out = torch.zeros(px.numel(), dtype=torch.complex128, device=px.device)
    for a, b in _blocks(px.numel(), fx.numel()):
        dx, dy = fx[a:b, None] - px[None, :], fy[a:b, None] - py[None, :]
        R = torch.sqrt(dx * dx + dy * dy + z * z)
        u, ph = 1.0 / R, k * R
        c, s = u * torch.cos(ph), u * torch.sin(ph)
        vr, vi = v.real[a:b], v.imag[a:b]
        out += torch.complex(vr @ c + vi @ s, vi @ c - vr @ s)
    return out


def _natural_spline(x, y):
    """Second derivatives of the natural cubic spline through (x, y)."""
    n, h = len(x), np.diff(x)
    A, r = np.eye(n), np.zeros(n)
    for i in range(1, n - 1):
        A[i, i - 1], A[i, i], A[i, i + 1] = h[i - 1] / 6, (h[i - 1] + h[i]) / 3, h[i] / 6
        r[i] = (y[i + 1] - y[i]) / h[i] - (y[i] - y[i - 1]) / h[i - 1]
    return np.linalg.solve(A, r)


def _spline_eval(x, y, m, u):
    """Value and derivative at u."""
    i = np.clip(np.searchsorted(x, u, side="right") - 1, 0, len(x) - 2)
    h, a, b = x[i + 1] - x[i], x[i + 1] - u, u - x[i]
    val = (m[i] * a ** 3 + m[i + 1] * b ** 3) / (6 * h) + (y[i] / h - m[i] * h / 6) * a + (y[i + 1] / h - m[i + 1] * h / 6) * b
    der = (-m[i] * a ** 2 + m[i + 1] * b ** 2) / (2 * h) - (y[i] / h - m[i] * h / 6) + (y[i + 1] / h - m[i + 1] * h / 6)
    return val, der


def _exact_far(case, seed):
    kind = case["kind"]
    ap, half = _aperture(case, seed)
    npix = case["nx"] * case["nz"] if kind == "zx" else case["n"] ** 2
    if float(ap.npil) * npix * (2 if kind == "design" else 1) > 1.5e11:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    px, py, t = (torch.tensor(a, device=dev) for a in (ap.px, ap.py, ap.t))
    z = torch.tensor(ap.focal_um, dtype=torch.float64, device=dev)
    k = 2.0 * math.pi / ap.wavelength_um
    if kind == "zx":
        nx, nz, f = case["nx"], case["nz"], ap.focal_um
        x = -half + 2 * half * torch.arange(nx, dtype=torch.float64, device=dev) / (nx - 1)
        zz = 0.8 * f + (1.2 * f - 0.8 * f) * torch.arange(nz, dtype=torch.float64, device=dev) / (nz - 1)
        fx, z = x.repeat(nz), zz.repeat_interleave(nx)
        E = _field64(px, py, t, fx, torch.zeros_like(fx), z, k)
        return (E.real ** 2 + E.imag ** 2).reshape(nz, nx).cpu().numpy()
    n = case["n"]
    x = -half + torch.arange(n, dtype=torch.float64, device=dev) * (2.0 * half / (n - 1))
    fx, fy = x.repeat(n), x.repeat_interleave(n)
    if kind != "design":
        E = _field64(px, py, t, fx, fy, z, k).reshape(n, n)
        inten = E.real ** 2 + E.imag ** 2
        return inten.cpu().numpy() if kind == "psf_host" else (E, inten)
    fill, amp, phase = _spline_tables()
    w = _fills(case, seed, ap.npil)
    A, dA = _spline_eval(fill, amp, _natural_spline(fill, amp), w)
    P, dP = _spline_eval(fill, phase, _natural_spline(fill, phase), w)
    t = torch.tensor(A * np.exp(1j * P), device=dev)
    E = _field64(px, py, t, fx, fy, z, k)
    inten = E.real ** 2 + E.imag ** 2
    mask = (fx ** 2 + fy ** 2 <= 1.0).to(torch.float64)
    inside, total = (inten * mask).sum(), inten.sum()
    gE = 2.0 * E * (inside / total ** 2 - mask / total)
    g = _adjoint64(px, py, gE, fx, fy, z, k).cpu().numpy()
    e = np.exp(1j * P)
    return E.reshape(n, n), -inside / total, np.real(np.conj(g) * (dA + 1j * A * dP) * e)


def _sinc(m, fill):
    return np.where(m == 0, fill, np.sin(np.pi * m * fill) / (np.pi * np.where(m == 0, 1, m)))


def _eps_operators(c, p, q, M):
    """(1/eps), Exx, Eyy over the orders: analytic rectangle with the inverse rule,
    or the Laurent rule on a 4 x 4 supersampled raster."""
    ep, eb, fx = c["eps_pillar"], c["eps_bg"], c["fill_x"]
    fy = c.get("fill_y", fx)
    dp, dq = p[:, None] - p[None, :], q[:, None] - q[None, :]
    if not c.get("force_laurent"):
        d = 1.0 / ep - 1.0 / eb
        a = np.arange(-M, M + 1)
        hx = np.linalg.inv(np.eye(2 * M + 1) / eb + d * _sinc(a[:, None] - a[None, :], fx))
        hy = np.linalg.inv(np.eye(2 * M + 1) / eb + d * _sinc(a[:, None] - a[None, :], fy))
        sx, sy = _sinc(dp, fx), _sinc(dq, fy)
        einv = d * sx * sy + np.eye(len(p)) / eb
        exx = hx[p[:, None] + M, p[None, :] + M] * sy + np.where(dp == 0, eb * ((dq == 0) - sy), 0.0)
        eyy = hy[q[:, None] + M, q[None, :] + M] * sx + np.where(dq == 0, eb * ((dp == 0) - sx), 0.0)
        return einv, exx, eyy
    ng = c["grid"] if c["grid"] > 0 else max(128, 8 * (2 * M + 1))
    s = (np.arange(ng)[:, None] + (np.arange(4)[None, :] + 0.5) / 4) / ng - 0.5
    s = s.reshape(-1)
    if c["shape"] == capi.SHAPE_RECT:
        inside = (np.abs(s)[:, None] <= fy * 0.5) & (np.abs(s)[None, :] <= fx * 0.5)
    else:
        r2 = ((s / (fy * 0.5)) ** 2)[:, None] + ((s / (fx * 0.5)) ** 2)[None, :]
        inside = (r2 <= 1.0) & ((c["shape"] == capi.SHAPE_ELLIPSE) | (r2 >= c["shape_param"] ** 2))
    eps = eb + (ep - eb) * inside.reshape(ng, 4, ng, 4).sum(axis=(1, 3)) / 16.0
    m = np.arange(-2 * M, 2 * M + 1)
    ph = np.exp(-2j * np.pi * m[:, None] * ((np.arange(ng) + 0.5) / ng - 0.5)[None, :]) / ng
    G = (ph @ eps @ ph.T).T
    T = G[dp + 2 * M, dq + 2 * M]
    return np.linalg.inv(T), T, T


def _rcwa64(layers, M):
    """X and Y results of one stack: rows (R, T, sum_de, de_t0, de_r0, tx0, ty0)."""
    c0 = layers[0]
    a = np.arange(-M, M + 1)
    p, q = np.repeat(a, 2 * M + 1), np.tile(a, 2 * M + 1)
    N, w = len(p), 2 * np.pi / c0["wavelength_um"]
    th, phi, n_inc, n_sub = c0.get("theta_rad", 0.0), c0.get("phi_rad", 0.0), c0["n_inc"], c0["n_sub"]
    kx = n_inc * math.sin(th) * math.cos(phi) * w - 2 * np.pi * p / c0.get("period_x_um", c0["period_um"])
    ky = n_inc * math.sin(th) * math.sin(phi) * w - 2 * np.pi * q / c0.get("period_y_um", c0["period_um"])
    J = np.vstack([-np.diag(ky), np.diag(kx)])
    K = np.vstack([np.diag(kx), np.diag(ky)])
    up = lambda v: np.where(v.imag < 0, -v, v)  # noqa: E731

    def half_space(n):
        kz = up(np.sqrt(n * n * w * w - kx * kx - ky * ky + 0j))
        kp = w * w * np.eye(2 * N) - J @ J.T / (n * n)
        return np.concatenate([kz, kz]), np.eye(2 * N), kp, 0.0

    def patterned(c):
        einv, exx, eyy = _eps_operators(c, p, q, M)
        kp = w * w * np.eye(2 * N) - J @ einv @ J.T
        e2 = np.zeros((2 * N, 2 * N), complex)
        e2[:N, :N], e2[N:, N:] = eyy, exx
        lam, W = np.linalg.eig(e2 @ kp - K @ K.T)
        return up(np.sqrt(lam + 0j)), W, kp, c["thickness_um"]

    regions = [half_space(n_inc)] + [patterned(c) for c in layers] + [half_space(n_sub)]
    i0 = M * (2 * M + 1) + M
    a0 = np.zeros((2 * N, 2), complex)
    a0[N + i0, 0], a0[i0, 1] = 1.0, -1.0
    s11, s12, s21, s22 = a0.copy(), np.zeros((2 * N, 2 * N), complex), np.zeros((2 * N, 2), complex), np.eye(2 * N, dtype=complex)
    for (qa, Wa, ka, ha), (qb, Wb, kb, hb) in zip(regions[:-1], regions[1:]):
        Q = np.linalg.solve(Wa, Wb)
        P = qa[:, None] * np.linalg.solve(ka @ Wa, kb @ Wb) / qb[None, :]
        t11, t12 = 0.5 * (Q + P), 0.5 * (Q - P)
        d1, d2 = np.exp(1j * qa * ha)[:, None], np.exp(1j * qb * hb)[None, :]
        X = t11 - d1 * (s12 @ t12)
        s12n = np.linalg.solve(X, d1 * (s12 @ t11) - t12) * d2
        s11 = np.linalg.solve(X, d1 * s11)
        s21 = s21 + s22 @ (t12 @ s11)
        s22 = s22 @ (t12 @ s12n + t11 * d2)
        s12 = s12n
    rows = []
    for e in range(2):
        def fields(region, v):
            return (region[2] @ (region[1] @ (v / (w * region[0]))))

        aN, b0 = s11[:, e], s21[:, e]
        Ha, Hb, Ht = fields(regions[0], a0[:, e]), fields(regions[0], b0), fields(regions[-1], aN)
        norm = n_inc / math.cos(th)
        diff = 0.5 * (np.conj(b0) * Ha - np.conj(Hb) * a0[:, e])
        bwd = (-(np.conj(Hb) * b0).real + diff.conj()).real
        fwd = (np.conj(Ht) * aN).real
        r, t = -(bwd[:N] + bwd[N:]) * norm, (fwd[:N] + fwd[N:]) * norm
        inc = Ha[N + i0] if abs(Ha[N + i0]) > 1e-30 else 1.0
        rows.append((r.sum(), t.sum(), r.sum() + t.sum(), t[i0], r[i0], Ht[N + i0] / inc, -Ht[i0] / inc))
    return rows


def exact(case, seed):
    if case["kind"] in ("psf_host", "psf", "zx", "design"):
        return _exact_far(case, seed)
    cells, nl = _cells(case, seed), case.get("layers", 1)
    # dense eigensolves on the host: this bound keeps them within a few seconds
    if sum((2.0 * (2 * c["Mx"] + 1) ** 2) ** 3 for c in cells) > 6e8:
        return None
    rows = []
    for i in range(0, len(cells), nl):
        rows += _rcwa64(cells[i:i + nl], cells[i]["Mx"])
    if case["kind"] == "cell":
        return np.array(rows[:1])
    return np.array(rows), None
