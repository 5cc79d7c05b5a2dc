"""Workloads of the engine, through its Python binding (``varrcwa_b200.capi``).

A case names an entry point (``call``), a structure family and its sizes:

``powers``  ``Context.order_powers``: per-order reflected / transmitted power of
            cells between two half-spaces, by adaptive varRCWA or plain RCWA.
``cells``   ``Context.redheffer`` or ``Context.differential``: the S-matrix
            blocks of cells, carried over to the Fourier basis of the E field
            as a caller does that joins them to another solver's blocks
            (eigenvector order, phase and mixing belong to the solver).
``stacks``  ``Context.stack_forward`` and ``stack_backward``: one optimisation
            step of freeform metagratings, per-order powers and the gradients
            with respect to every pixel and every layer thickness.
``knots``   ``Context.redheffer_forward`` and ``redheffer_backward``: one
            optimisation step of waveguide mode converters, the blocks and the
            gradient with respect to the width control points.

Sizes are the ones of the benchmark configurations and of the tests (5 x 5 to
15 x 15 orders in two dimensions, 15 to 41 in one).  Pillars sit in a
rectangular lattice: on a square one modes are exactly degenerate, and which
basis of a degenerate pair a solver's rounding picks decides whether a segment
is split.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from varrcwa_b200 import capi, objectives, structures

_CONTEXTS = {}


def _context():
    """The engine context of this process (a program keeps one per device)."""
    if 0 not in _CONTEXTS:
        _CONTEXTS[0] = capi.Context(0)
    return _CONTEXTS[0]


def listed():
    return [
        # one lamellar grating, one slice: the smallest call, an interactive single solve
        dict(name="grating_21_single", call="powers", family="grating", nx=21, ny=1, batch=1, method="rcwa", slices=1),
        # one short 2D taper at the 41 orders of the taper benchmark: thousands of small batched products
        dict(name="taper_41", call="cells", family="taper", nx=41, ny=1, batch=1, method="redheffer", pe=1e-4,
             length=1.0),
        # one 7 x 7 pillar: the latency of a single adaptive solve
        dict(name="pillar_7_single", call="powers", family="pillar", nx=7, ny=7, batch=1, method="redheffer", pe=1e-2),
        # a sweep of pillars at 11 x 11 orders, the usual unit-cell library
        dict(name="pillars_11_b16", call="powers", family="pillar", nx=11, ny=11, batch=16, method="redheffer",
             pe=1e-2),
        # a mixed queue of pillars, 7 x 7 to 15 x 15 orders in one call
        dict(name="pillars_mixed_b8", call="powers", family="pillar_mixed", nx=15, ny=15, batch=8,
             method="redheffer", pe=1e-2),
        # sixteen slices of a pillar by plain RCWA, the conventional check of an adaptive solve
        dict(name="pillar_13x9_rcwa", call="powers", family="pillar", nx=13, ny=9, batch=2, method="rcwa", slices=16),
        # differential method on rectangular cells with a moving edge
        dict(name="edge_9x7_differential", call="cells", family="edge", nx=9, ny=7, batch=4, method="differential",
             slices=8),
        # a planar (layout) taper between PML, the photonic-circuit path
        dict(name="planar_11x5", call="cells", family="planar", nx=11, ny=5, batch=1, method="redheffer", pe=1e-2,
             length=1.0),
        # one metagrating of the freeform optimisation: forward and gradients
        dict(name="metagrating_9_single", call="stacks", nx=9, ny=9, batch=1, layers=4, npix=64),
        # a population of metagratings per optimisation step
        dict(name="metagratings_9_b32", call="stacks", nx=9, ny=9, batch=32, layers=4, npix=64),
        # the same at 15 x 15 orders, n = 450
        dict(name="metagratings_15_b4", call="stacks", nx=15, ny=15, batch=4, layers=4, npix=64),
        # mode converters between PML: forward and gradient of the width control points
        dict(name="converter_7_knots", call="knots", nx=7, ny=7, batch=1, pe=1e-2, length=0.6),
    ]


def draw(rng):
    """One more case of the same ranges: odd harmonic counts, batches from one up."""

    def odd(lo, hi):
        return 2 * int(round((math.exp(rng.uniform(math.log(lo), math.log(hi))) - 1) / 2)) + 1

    def batch_for(n, most):
        # no more than the mixed queue's work: its largest cells are n = 450
        cap = max(1, min(most, int(4 * (300.0 / n) ** 3)))
        return int(round(math.exp(rng.uniform(0.0, math.log(cap + 0.49)))))

    kind = rng.choice(["grating", "taper", "pillar", "pillar", "rcwa", "edge", "planar", "stacks", "stacks", "knots"])
    if kind == "grating":
        return dict(call="powers", family="grating", nx=odd(11, 61), ny=1, batch=rng.randint(1, 8), method="rcwa",
                    slices=rng.randint(1, 3))
    if kind == "taper":
        return dict(call="cells", family="taper", nx=odd(21, 51), ny=1, batch=rng.randint(1, 3), method="redheffer",
                    pe=10.0 ** rng.uniform(-4.0, -2.5), length=rng.uniform(0.4, 1.0))
    if kind == "planar":
        return dict(call="cells", family="planar", nx=odd(9, 13), ny=odd(3, 7), batch=1, method="redheffer",
                    pe=10.0 ** rng.uniform(-2.0, -1.3), length=rng.uniform(0.4, 1.0))
    if kind == "knots":
        return dict(call="knots", nx=odd(5, 7), ny=odd(5, 7), batch=rng.randint(1, 2), pe=10.0 ** rng.uniform(-2.0, -1.3),
                    length=rng.uniform(0.2, 0.5))
    nx, ny = odd(5, 15), odd(5, 15)
    n = 2 * nx * ny
    if kind == "stacks":
        return dict(call="stacks", nx=nx, ny=ny, batch=batch_for(n, 40), layers=rng.randint(1, 4),
                    npix=rng.choice([32, 48, 64]))
    if kind == "edge":
        return dict(call="cells", family="edge", nx=nx, ny=ny, batch=batch_for(n, 6), method="differential",
                    slices=rng.randint(2, 8))
    if kind == "rcwa":
        return dict(call="powers", family="pillar", nx=nx, ny=ny, batch=batch_for(n, 4), method="rcwa",
                    slices=rng.randint(2, 12))
    return dict(call="powers", family="pillar", nx=nx, ny=ny, batch=batch_for(n, 20), method="redheffer",
                pe=10.0 ** rng.uniform(-2.3, -1.7))


# ---------------------------------------------------------------------------
# Structures (seeded)
# ---------------------------------------------------------------------------
def _pillar(rng, nx, ny):
    d = structures.pillar_cell(int(rng.integers(1 << 30)), norders=11, lam=float(rng.uniform(0.45, 0.65)))
    d.update(nx=nx, ny=ny, Lx=float(rng.uniform(0.38, 0.42)), Ly=float(rng.uniform(0.43, 0.47)))
    return d


def _cells(case, seed):
    rng = np.random.default_rng([77, int(seed)])
    out = []
    for k in range(case["batch"]):
        nx, ny, fam = case["nx"], case["ny"], case["family"]
        if fam == "pillar":
            d = _pillar(rng, nx, ny)
        elif fam == "pillar_mixed":  # 7 x 7 up to nx x nx
            o = 7 + 2 * (k % ((nx - 7) // 2 + 1))
            d = _pillar(rng, o, o)
        elif fam == "grating":
            a = rng.uniform(0.1, 0.4)
            b = a + rng.uniform(0.2, 0.5)
            d = dict(kind="grid", lam=float(rng.uniform(1.3, 1.7)), nx=nx, ny=ny, pml=False,
                     x=np.array([0.0, a, b, 1.0]), y=np.array([0.0, 1.0]),
                     eps=np.array([[2.085, 12.11, 2.085]], dtype=np.complex128), z0=0.0,
                     z1=float(rng.uniform(0.2, 0.6)), end0=2.085, end1=1.0)
        elif fam == "taper":
            w0 = rng.uniform(0.35, 0.45)
            d = structures.taper_2d(norders=nx, length=case["length"], w0=w0, w1=w0 + 0.06 * case["length"])
        elif fam == "planar":
            w0 = rng.uniform(0.45, 0.6)
            d = structures.planar_taper(w0=w0, w1=w0 + 0.18 * case["length"], length=case["length"],
                                        norders=(nx, ny))
        elif fam == "edge":
            e = rng.uniform(0.38, 0.46)
            d = dict(kind="grid", lam=float(rng.uniform(1.2, 1.4)), nx=nx, ny=ny, pml=False,
                     x=np.array([0.0, 0.13, e, 0.62, 1.0]), y=np.array([0.0, 0.21, 0.35, 0.8]),
                     eps=np.array([[2.085, 2.085, 2.085, 2.085], [2.085, 12.11, 4.0, 2.085],
                                   [2.085, 2.085, 2.085, 2.085]], dtype=np.complex128),
                     xrules=[(2, [0.0, 0.2], [e, e + 0.1])], z0=0.0, z1=0.2, end0=2.085, end1=1.0)
        else:
            raise ValueError(fam)
        out.append(d)
    return out


def _stacks(case, seed):
    rng = np.random.default_rng([78, int(seed)])
    out = []
    for _ in range(case["batch"]):
        d = structures.metagrating_c4(int(rng.integers(1 << 30)), npix=case["npix"], nlayers=case["layers"])
        d.update(nx=case["nx"], ny=case["ny"])
        out.append(d)
    m = case["nx"] * case["ny"]
    w = rng.uniform(0.0, 1.0, (2, case["batch"], m))
    return out, w[0], w[1]


def _converters(case, seed):
    rng = np.random.default_rng([79, int(seed)])
    out = []
    for _ in range(case["batch"]):
        # a part of the 20 um converter with its control point spacing
        d = structures.waveguide_pml(int(rng.integers(1 << 30)), norders=case["nx"], ncontrol=5,
                                     length=case["length"], spline=True)
        w = 0.6 + 0.25 * (d["widths"] - 0.75) * case["length"]
        d["xrules"] = [(i, zs, 2.0 + s * 0.5 * w) for (i, zs, _), s in zip(d["xrules"], (-1.0, 1.0))]
        d.update(ny=case["ny"], widths=w)
        out.append(d)
    return out


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    state = dict(case=case, ctx=_context())
    if case["call"] == "stacks":
        state["stacks"], state["wR"], state["wT"] = _stacks(case, seed)
    elif case["call"] == "knots":
        state["cells"] = _converters(case, seed)
    else:
        state["cells"] = _cells(case, seed)
    return state


def _fourier(r):
    w0i, w1i = np.linalg.inv(r["W0"]), np.linalg.inv(r["W1"])
    return dict(Tuu=r["W1"] @ r["Tuu"] @ w0i, Tdd=r["W0"] @ r["Tdd"] @ w1i, Rdu=r["W0"] @ r["Rdu"] @ w0i,
                Rud=r["W1"] @ r["Rud"] @ w1i)


def run(state):
    case, ctx = state["case"], state["ctx"]
    if case["call"] == "powers":
        out = ctx.order_powers(state["cells"], method=case["method"], pe=case.get("pe", 1e-2),
                               nslices=case.get("slices", 1), side=1)
        return dict(R=np.concatenate([o["R"].ravel() for o in out]), T=np.concatenate([o["T"].ravel() for o in out]),
                    status=np.array([o["status"] for o in out]))
    if case["call"] == "cells":
        if case["method"] == "redheffer":
            out = ctx.redheffer(state["cells"], pe=case["pe"])
        else:
            out = ctx.differential(state["cells"], case["slices"])
        return [dict(_fourier(r), N=r["N"], status=r["status"]) for r in out]
    if case["call"] == "stacks":
        ref, trn, status = ctx.stack_forward(state["stacks"])
        g, gt = ctx.stack_backward(state["wR"], state["wT"], want_thick=True)
        return dict(REF=ref, TRN=trn, grad=g, grad_thick=gt, status=status)
    res = ctx.redheffer_forward(state["cells"], pe=case["pe"])
    gS, gB = [], []
    for r in res:
        i0, i1 = int(np.argmax(r["gam0"].real)), int(np.argmax(r["gam1"].real))
        _, s, b = objectives.mode_conversion(r, i0, i1)
        gS.append(s)
        gB.append(b)
    grads = ctx.redheffer_backward(gS, gB)
    return [dict(_fourier(r), N=r["N"], status=r["status"], grad=np.stack(g)) for r, g in zip(res, grads)]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Nominal FP64 operations of the method (LAPACK counts, real operations:
    an eigen-decomposition with its inverses 121 n^3, a perturbative segment
    and its star product 293 n^3, an assembled sample 12 n^3) and the bytes of
    the inputs and results.  An adaptive solve is counted with one rejected
    root and three accepted segments, which most of these structures exceed."""
    B = case["batch"]
    if case.get("family") == "pillar_mixed":
        orders = [7 + 2 * (k % ((case["nx"] - 7) // 2 + 1)) for k in range(B)]
        ns = [2 * o * o for o in orders]
    else:
        ns = [2 * case["nx"] * case["ny"]] * B
    if case["call"] == "stacks":
        eigs, segs, samples, outs = case["layers"], case["layers"], case["layers"], 0
        nbytes = B * (case["layers"] * case["npix"] ** 2 * 16.0 + 16.0 * ns[0])
    else:
        method = case.get("method", "redheffer")
        if method == "redheffer":
            eigs, segs, samples = 3, 3, 7
        elif method == "rcwa":
            eigs, segs, samples = case["slices"], case["slices"], case["slices"]
        else:
            eigs, segs, samples = 0, case["slices"], 2 * case["slices"] + 1
        outs = 4 if case["call"] != "powers" else 0
        nbytes = sum(16.0 * n + outs * 16.0 * n * n for n in ns)
    flops = sum((121.0 * eigs + 293.0 * segs + 12.0 * samples) * float(n) ** 3 for n in ns)
    if case["call"] in ("stacks", "knots"):
        flops *= 2.0  # the reverse pass costs at least the forward's products
    return dict(bytes=nbytes, flops=flops)


# ---------------------------------------------------------------------------
# The same values from plain torch on the CPU, in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    n = 2 * case["nx"] * case["ny"]
    if case["call"] == "stacks":
        if case["batch"] * case["layers"] * (n / 162.0) ** 3 > 12:
            return None
        return _exact_stacks(case, seed)
    if case["call"] == "knots":  # the gradient is that of the frozen segmentation: no closed value
        cells = _converters(case, seed)
    else:
        cells = _cells(case, seed)
    cost = {"grating": 0.05, "edge": 0.05, "taper": 60.0, "planar": 60.0}.get(case.get("family"), 12.0)
    if case.get("method") == "rcwa":
        cost = 1.2 * case["slices"]
    if case["batch"] * cost * (n / 162.0) ** 3 > 40:
        return None
    out = []
    for d in cells:
        with torch.no_grad():
            s = _solve(d, case)
            if case["call"] == "powers":
                out.append(_powers(d, s))
                continue
            r = _to_fourier(s)
            r.update(N=None, status=None)
            if case["call"] == "knots":
                r["grad"] = None
            out.append(r)
    if case["call"] == "powers":
        return dict(R=np.concatenate([r.ravel() for r, _ in out]), T=np.concatenate([t.ravel() for _, t in out]),
                    status=None)
    return out


_C = torch.complex128


def _edges(x, count):
    """Fourier coefficients of the indicator of [x[j], x[j+1]], harmonics -(count-1)/2 .. : count x cells."""
    x = torch.as_tensor(np.asarray(x, dtype=np.float64))
    h = torch.arange(count, dtype=torch.float64)[:, None] - (count - 1) // 2
    d, w, mid = x[-1] - x[0], (x[1:] - x[:-1])[None], (0.5 * (x[1:] + x[:-1]))[None]
    return torch.sinc(h * w / d) * (w / d) * torch.exp(-2j * math.pi * h * mid / d)


def _toeplitz(v):
    """Toeplitz matrices of the last axis: v[..., n-1 + r - c]."""
    n = (v.shape[-1] + 1) // 2
    i = torch.arange(n)
    return v[..., n - 1 + i[:, None] - i[None, :]]


def _convolutions(x, y, eps, nx, ny):
    """fe11, fe22 (inverse rule across x / across y) and fe33 of a raster eps (y strips x x cells)."""
    ex, ey = _edges(x, 2 * nx - 1), _edges(y, 2 * ny - 1)
    m = nx * ny
    inv = 1.0 / eps
    tx = torch.linalg.inv(_toeplitz(inv @ ex.T))  # strips x nx x nx
    fe11 = torch.einsum("sik,sjl->ijkl", tx, _toeplitz(ey.T)).reshape(m, m)
    ty = torch.linalg.inv(_toeplitz(inv.T @ ey.T))  # cells x ny x ny
    fe22 = torch.einsum("cik,cjl->ijkl", _toeplitz(ex.T), ty).reshape(m, m)
    f = ex @ eps.T @ ey.T
    i, j = torch.arange(nx), torch.arange(ny)
    fe33 = f[(nx - 1 + i[:, None] - i[None, :])[:, None, :, None], (ny - 1 + j[:, None] - j[None, :])[None, :, None, :]]
    return fe11, fe22, fe33.reshape(m, m)


def _stretch(x, count):
    """Fourier coefficients of the PML stretch s(x): 1 inside, the
    coordinate-transform profile (1 - gamma sin^2) cos^2 in the outer cells,
    gamma = 1 / (1 - i), and of the unit profile."""
    L, gam = float(x[-1] - x[0]), 1.0 / (1.0 - 1.0j)
    h = np.arange(count) - (count - 1) // 2

    def layer(b0, b1, sign):
        bm, bp = (b1 - b0) / L, (b1 + b0) / L
        r = 4.0 * np.sinc(h * bm - 0.5) * np.exp(-1j * np.pi * (h * bp + sign * 0.5))
        r = r + (8.0 - 2.0 * gam) * np.sinc(h * bm) * np.exp(-1j * np.pi * h * bp)
        r = r + 4.0 * np.sinc(h * bm + 0.5) * np.exp(-1j * np.pi * (h * bp - sign * 0.5))
        r = r + gam * np.sinc(h * bm - 1.0) * np.exp(-1j * np.pi * (h * bp + sign))
        r = r + gam * np.sinc(h * bm + 1.0) * np.exp(-1j * np.pi * (h * bp - sign))
        return r * bm / 16.0

    a, b = float(x[1]), float(x[-2])
    return (b - a) / L * np.sinc(h * (b - a) / L) * np.exp(-1j * np.pi * h * (a + b) / L) + layer(x[0], a, 1.0) + \
        layer(b, x[-1], -1.0)


def _wavevectors(d, x, y):
    nx, ny = d["nx"], d["ny"]
    ax = 2 * math.pi / (x[-1] - x[0]) * (np.arange(nx) - nx // 2)
    ay = 2 * math.pi / (y[-1] - y[0]) * (np.arange(ny) - ny // 2)
    kx, ky = torch.diag(torch.as_tensor(ax)).to(_C), torch.diag(torch.as_tensor(ay)).to(_C)
    if d["pml"]:
        kx = _toeplitz(torch.as_tensor(_stretch(x, 2 * nx - 1))) @ kx
        ky = _toeplitz(torch.as_tensor(_stretch(y, 2 * ny - 1))) @ ky
    return torch.kron(kx, torch.eye(ny, dtype=_C)), torch.kron(torch.eye(nx, dtype=_C), ky)


def _section(d, z):
    """x, y, eps of a structure at z."""
    if d["kind"] == "planar":
        (pts,) = d["polys"]
        k = len(pts)
        cross = []
        for i in range(k):
            (x0, z0), (x1, z1) = pts[i], pts[(i + 1) % k]
            if z0 <= z < z1 or z1 <= z < z0:
                cross.append(x0 + (z - z0) / (z1 - z0) * (x1 - x0))
        return d["frame"](sorted(cross))
    x, y, eps = _geometry(d, z)
    return x, y, torch.as_tensor(eps).to(_C)


def _geometry(d, z):
    """Coordinates and permittivity at z (linear or natural cubic spline rules, pillar raster)."""
    if d["kind"] == "pillar":
        n, r = d["npx"], d["r0"] + (d["r1"] - d["r0"]) * (z - d["z0"]) / (d["z1"] - d["z0"])
        cx = (np.arange(n) + 0.5) * (d["Lx"] / n) - 0.5 * d["Lx"]
        cy = (np.arange(n) + 0.5) * (d["Ly"] / n) - 0.5 * d["Ly"]
        eps = np.where(cx[None] ** 2 + cy[:, None] ** 2 <= r * r, d["eps_in"], d["eps_out"])
        return np.linspace(0.0, d["Lx"], n + 1), np.linspace(0.0, d["Ly"], n + 1), eps
    x, y = np.array(d["x"], dtype=np.float64), np.array(d["y"], dtype=np.float64)
    for i, zs, v in d.get("xrules", []):
        x[i] = _spline(zs, v, z) if d.get("spline") else np.interp(z, zs, v)
    return x, y, d["eps"]


def _spline(zs, v, z):
    zs, v = np.asarray(zs, dtype=np.float64), np.asarray(v, dtype=np.float64)
    if z <= zs[0] or z >= zs[-1]:
        return float(v[0] if z <= zs[0] else v[-1])
    h, k = np.diff(zs), len(zs)
    A, r = np.eye(k), np.zeros(k)
    for i in range(1, k - 1):
        A[i, i - 1:i + 2] = h[i - 1], 2 * (h[i - 1] + h[i]), h[i]
        r[i] = 6 * ((v[i + 1] - v[i]) / h[i] - (v[i] - v[i - 1]) / h[i - 1])
    M = np.linalg.solve(A, r)
    i = int(np.searchsorted(zs, z, side="right")) - 1
    a, b = (zs[i + 1] - z) / h[i], (z - zs[i]) / h[i]
    return float(a * v[i] + b * v[i + 1] + ((a ** 3 - a) * M[i] + (b ** 3 - b) * M[i + 1]) * h[i] ** 2 / 6)


def _operators(d, sec, K):
    x, y, eps = sec
    kx, ky = K
    fe11, fe22, fe33 = _convolutions(x, y, eps, d["nx"], d["ny"])
    k2 = (2 * math.pi / d["lam"]) ** 2
    one = k2 * torch.eye(kx.shape[0], dtype=_C)
    ix, iy = torch.linalg.solve(fe33, kx), torch.linalg.solve(fe33, ky)
    P = torch.cat([torch.cat([kx @ iy, one - kx @ ix], 1), torch.cat([ky @ iy - one, -ky @ ix], 1)])
    Q = torch.cat([torch.cat([-kx @ ky, kx @ kx - k2 * fe22], 1), torch.cat([k2 * fe11 - ky @ ky, ky @ kx], 1)])
    return P, Q


def _branch(lam):
    """Square root with a decaying or forward-going sign."""
    g = torch.sqrt(lam)
    g = torch.where(g.imag < 0, -g, g)
    return torch.where((g.imag.abs() < g.real.abs()) & (g.real < 0), -g, g)


def _modes(P, Q):
    lam, W = torch.linalg.eig(P @ Q)
    g = _branch(lam)
    return W, Q @ W / g, g


def _halfspace(d, eps, K):
    """Plane waves of a homogeneous medium: W = I."""
    kx, ky = (torch.diagonal(k) for k in K)
    k2 = (2 * math.pi / d["lam"]) ** 2
    g = _branch(k2 * (k2 * eps - kx * kx - ky * ky))
    V = torch.cat([torch.cat([torch.diag(-kx * ky / g), torch.diag((kx * kx - k2 * eps) / g)], 1),
                   torch.cat([torch.diag((k2 * eps - ky * ky) / g), torch.diag(kx * ky / g)], 1)])
    return torch.eye(2 * len(kx), dtype=_C), V, torch.cat([g, g])


def _join(S, left, right):
    """S (ending in modes `left`) continued across the interface into modes `right`."""
    f, h = torch.linalg.solve(left[0], right[0]), torch.linalg.solve(left[1], right[1])
    A, B = 0.5 * (f + h), 0.5 * (f - h)
    Ai = torch.linalg.inv(A)
    return _star(S, (A - B @ Ai @ B, Ai, -Ai @ B, B @ Ai))


def _star(S, s):
    Tdd, Tuu, Rud, Rdu = S
    tdd, tuu, rud, rdu = s
    one = torch.eye(Tdd.shape[0], dtype=_C)
    a = torch.linalg.solve(one - rdu @ Rud, torch.cat([tdd, rdu @ Tuu], 1))
    a, b = a[:, :len(one)], a[:, len(one):]
    return Tdd @ a, tuu @ (Tuu + Rud @ b), rud + tuu @ Rud @ a, Rdu + Tdd @ b


def _uniform(mode, t):
    X = torch.diag(torch.exp(1j * mode[2] * t))
    return X, X, torch.zeros_like(X), torch.zeros_like(X)


def _segment(P0, mode, k0, dz, ends):
    """Simpson's rule for the first-order perturbation of a segment by its end and mid samples."""
    W, V, g = mode
    dA, dB = [], []
    for P, Q in ends:
        u, v = torch.linalg.solve(W, (P - P0[0]) @ V), torch.linalg.solve(V, (Q - P0[1]) @ W)
        dA.append(u + v)
        dB.append(u - v)
    h, f, c = torch.exp(0.5j * dz / k0 * g), torch.exp(1j * dz / k0 * g), 1j * dz / (12 * k0)
    (a0, a1), (b0, b1) = dA, dB
    tuu = c * (f[:, None] * a0 + a1 * f[None])
    tdd = c * (a0 * f[None] + f[:, None] * a1)
    rud = -c * (f[:, None] * b0 * f[None] + b1)
    rdu = -c * (b0 + f[:, None] * b1 * f[None])
    err = max(float(t.abs().max()) for t in (tuu, tdd, rud, rdu))
    return (tdd + torch.diag(f), tuu + torch.diag(f), rud, rdu), err


def _planar_frame(d):
    """Completes a planar cell: x from the crossings at z between spacers and PML, five y strips."""
    xs = [p[0] for p in d["polys"][0]]
    lo, hi = min(xs), max(xs)
    l, r, b, t = d["pml_w"]
    sl, sr, sb, st = d["space"]
    ys = np.cumsum([0.0, b, sb, d["thickness"], st, t])

    def frame(cross):
        x = np.array([lo - sl - l, lo - sl] + list(cross) + [hi + sr, hi + sr + r])
        eps = np.full((5, len(x) - 1), d["eps_bg"], dtype=np.complex128)
        eps[2, 2:-2:2] = d["eps_dev"]
        return x, ys, torch.as_tensor(eps)

    return frame


def _solve(d, case):
    """(entrance modes, exit modes, S) of a cell by the case's method."""
    if d["kind"] == "planar":
        d = dict(d, frame=_planar_frame(d))
    z0, z1, k0 = d["z0"], d["z1"], 2 * math.pi / d["lam"]
    x, y, _ = _section(d, 0.5 * (z0 + z1))
    K = _wavevectors(d, x, y)
    known = {}

    def at(z):
        if z not in known:
            known[z] = _operators(d, _section(d, z), K)
        return known[z]

    e0 = _halfspace(d, d["end0"], K) if d.get("end0") is not None else _modes(*at(z0))
    e1 = _halfspace(d, d["end1"], K) if d.get("end1") is not None else _modes(*at(z1))
    one = torch.eye(K[0].shape[0] * 2, dtype=_C)
    S, left = (one, one, torch.zeros_like(one), torch.zeros_like(one)), e0
    method = case.get("method", "redheffer")
    if method == "rcwa":
        dz = (z1 - z0) / case["slices"]
        for i in range(case["slices"]):
            mode = _modes(*at(z0 + (i + 0.5) * dz))
            S, left = _star(_join(S, left, mode), _uniform(mode, dz / k0)), mode
    elif method == "differential":
        dz = (z1 - z0) / case["slices"]
        S, left = _join(S, left, e1), e1
        for i in range(case["slices"]):
            S = _star(S, _propagator(e1, k0, dz, [at(z0 + (i + f) * dz) for f in (0.0, 0.5, 1.0)]))
    else:
        todo = [(z0, z1, None)]
        while todo:
            a, b, mode = todo.pop()
            zm = 0.5 * (a + b)
            mode = mode or (at(zm), _modes(*at(zm)))
            seg, err = _segment(mode[0], mode[1], k0, b - a, [at(a), at(b)])
            if err > case["pe"]:
                u, v = (2 * a + b) / 3, (a + 2 * b) / 3
                todo += [(v, b, None), (u, v, mode), (a, u, None)]
                continue
            S, left = _star(_join(S, left, mode[1]), seg), mode[1]
    return e0, e1, _join(S, left, e1)


def _propagator(mode, k0, dz, samples):
    """One slice of the differential method in the modes of the exit."""
    (P0, Q0), (P1, Q1), (P2, Q2) = samples
    W, V, _ = mode
    one = torch.eye(W.shape[0], dtype=_C)
    q = dz * dz / (k0 * k0)
    L11 = one - q / 6 * (P1 @ Q0 + P1 @ Q1 + P2 @ Q1 - q / 4 * P2 @ Q1 @ P1 @ Q0)
    L22 = one - q / 6 * (Q1 @ P0 + Q1 @ P1 + Q2 @ P1 - q / 4 * Q2 @ P1 @ Q1 @ P0)
    L12 = 1j * dz / (6 * k0) * (P0 + 4 * P1 + P2 - q / 2 * (P1 @ Q1 @ P0 + P2 @ Q1 @ P1))
    L21 = 1j * dz / (6 * k0) * (Q0 + 4 * Q1 + Q2 - q / 2 * (Q1 @ P1 @ Q0 + Q2 @ P1 @ Q1))
    f = torch.linalg.solve(W, torch.cat([L11 @ W, L12 @ V], 1))
    h = torch.linalg.solve(V, torch.cat([L21 @ W, L22 @ V], 1))
    n = len(one)
    up, dn = 0.5 * (f + h), 0.5 * (f - h)
    t11, t12 = up[:, :n] + up[:, n:], up[:, :n] - up[:, n:]
    t21, t22 = dn[:, :n] + dn[:, n:], dn[:, :n] - dn[:, n:]
    tdd = torch.linalg.inv(t22)
    rdu = -tdd @ t21
    return tdd, t11 + t12 @ rdu, t12 @ tdd, rdu


def _to_fourier(s):
    e0, e1, (Tdd, Tuu, Rud, Rdu) = s
    i0, i1 = torch.linalg.inv(e0[0]), torch.linalg.inv(e1[0])
    return {k: v.numpy() for k, v in dict(Tuu=e1[0] @ Tuu @ i0, Tdd=e0[0] @ Tdd @ i1, Rdu=e0[0] @ Rdu @ i0,
                                          Rud=e1[0] @ Rud @ i1).items()}


def _order_power(d, kx, ky, field, eps, norm):
    """Power per order of transverse harmonics `field` (2 m) in a homogeneous medium."""
    m, k0 = len(kx), 2 * math.pi / d["lam"]
    kz = torch.sqrt((k0 * k0 * eps - kx * kx - ky * ky).to(_C))
    ex, ey = field[:m], field[m:]
    ez = (kx * ex + ky * ey) / kz
    p = ex.abs() ** 2 + ey.abs() ** 2 + ez.abs() ** 2
    return kz.real.abs() * p / (math.sqrt(norm) * k0)


def _powers(d, s):
    """Incidence from the exit side, both polarisations."""
    e0, e1, (Tdd, _, Rud, _) = s
    x, y, _ = _section(d, d["z0"])
    kx, ky = (torch.diagonal(k).real for k in _wavevectors(d, x, y))
    m = len(kx)
    R, T = [], []
    for q in (0, m):
        c = q + d["ny"] * (d["nx"] // 2) + d["ny"] // 2
        R.append(_order_power(d, kx, ky, Rud[:, c], d["end1"], d["end1"]).numpy())
        T.append(_order_power(d, kx, ky, Tdd[:, c], d["end0"], d["end1"]).numpy())
    return np.stack(R), np.stack(T)


def _exact_stacks(case, seed):
    """Powers and their gradients by automatic differentiation of the stack's S-matrix."""
    stacks, wR, wT = _stacks(case, seed)
    out = dict(REF=[], TRN=[], grad=[], grad_thick=[])
    for d, wr, wt in zip(stacks, wR, wT):
        d = dict(d, pml=False)
        n = case["npix"]
        x, y = np.linspace(0.0, d["Lx"], n + 1), np.linspace(0.0, d["Ly"], n + 1)
        K = _wavevectors(d, x, y)
        k0 = 2 * math.pi / d["lam"]
        eps = torch.tensor(np.stack(d["layers"]), requires_grad=True)
        thick = torch.tensor(np.array(d["thick"], dtype=np.float64), requires_grad=True)
        e0, e1 = _halfspace(d, d["eps_in"], K), _halfspace(d, d["eps_out"], K)
        one = torch.eye(2 * K[0].shape[0], dtype=_C)
        S, left = (one, one, torch.zeros_like(one), torch.zeros_like(one)), e0
        for layer, t in zip(eps, thick):
            mode = _modes(*_operators(d, (x, y, layer.to(_C)), K))
            S, left = _star(_join(S, left, mode), _uniform(mode, t / k0)), mode
        _, Tuu, _, Rdu = _join(S, left, e1)
        kx, ky = (torch.diagonal(k).real for k in K)
        c = d["ny"] * (d["nx"] // 2) + d["ny"] // 2
        ref = _order_power(d, kx, ky, Rdu[:, c], d["eps_in"], d["eps_in"])
        trn = _order_power(d, kx, ky, Tuu[:, c], d["eps_out"], d["eps_in"])
        loss = (torch.as_tensor(wr) * ref).sum() + (torch.as_tensor(wt) * trn).sum()
        g, gt = torch.autograd.grad(loss, [eps, thick])
        for k, v in zip(("REF", "TRN", "grad", "grad_thick"), (ref.detach(), trn.detach(), g, gt)):
            out[k].append(v.numpy())
    return dict({k: np.stack(v) for k, v in out.items()}, status=None)
