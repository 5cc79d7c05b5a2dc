"""Order powers of mirror-symmetric cells through their parity classes against
the general way (VRC_NO_FOLD), to 1e-9 of the largest power as the other
order-power tests: every method, both sides, odd and equal harmonic counts,
single-row truncations, lossy media, odd rasters, mixed calls; same statuses
and the same trees (rectangular lattices: no degenerate modes)."""
import numpy as np
import pytest

from varrcwa_b200 import structures as st

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from varrcwa_b200.capi import Context
    c = Context(0)
    yield c
    c.close()


def _pillar(seed, nx, ny, npx=64, npy=64, **kw):
    d = st.pillar_cell(seed, norders=3, npix=npx, lam=0.55)
    d.update(nx=nx, ny=ny, npy=npy, Lx=0.41, Ly=0.46, **kw)
    return d


def _both(ctx, monkeypatch, cells, **kw):
    monkeypatch.delenv("VRC_NO_FOLD", raising=False)
    a = ctx.order_powers(cells, **kw)
    ta = [ctx.tree(c) for c in range(len(cells))]
    monkeypatch.setenv("VRC_NO_FOLD", "1")
    b = ctx.order_powers(cells, **kw)
    tb = [ctx.tree(c) for c in range(len(cells))]
    for c in range(len(cells)):
        assert a[c]["status"] == b[c]["status"] == 0
        for k in ("R", "T"):
            assert np.abs(a[c][k] - b[c][k]).max() <= 1e-9 * max(b[c]["R"].max(), b[c]["T"].max())
        assert [(x[0], x[1], x[3]) for x in ta[c]] == [(x[0], x[1], x[3]) for x in tb[c]]
    return a


@pytest.mark.parametrize("nx,ny", [(3, 3), (9, 1), (1, 9), (5, 3), (3, 7), (7, 5), (9, 9)])
@pytest.mark.parametrize("side", [0, 1])
def test_adaptive(ctx, monkeypatch, nx, ny, side):
    _both(ctx, monkeypatch, [_pillar(7, nx, ny)], method="redheffer", pe=1e-2, side=side)


@pytest.mark.parametrize("method", ["rcwa", "differential"])
@pytest.mark.parametrize("nx,ny", [(5, 3), (7, 7)])
def test_fixed_slices(ctx, monkeypatch, method, nx, ny):
    n = 4 if method == "rcwa" else 16
    for flux in (True, False):
        _both(ctx, monkeypatch, [_pillar(8, nx, ny, z1=0.1)], method=method, nslices=n, side=1, flux_norm=flux)


def test_lossy_and_odd_rasters(ctx, monkeypatch):
    _both(ctx, monkeypatch, [_pillar(9, 7, 5, npx=33, npy=64, eps_in=5.8 + 0.4j),
                             _pillar(10, 5, 7, npx=64, npy=31, eps_out=1.7 + 0.01j)], method="redheffer", pe=1e-2)


def test_mixed_call(ctx, monkeypatch):
    """Pillars of several truncations beside a grid cell, over the lanes."""
    g = dict(kind="grid", lam=1.3, nx=5, ny=3, pml=False, x=np.array([0.0, 0.13, 0.41, 1.0]),
             y=np.array([0.0, 0.3, 0.8]), eps=np.array([[2.0, 9.0, 2.0], [2.0, 2.0, 2.0]], dtype=complex),
             z0=0.0, z1=0.3, end0=2.085, end1=1.0)
    cells = [_pillar(20, 3, 3), g, _pillar(21, 5, 5), _pillar(22, 1, 1), _pillar(23, 7, 3), g, _pillar(24, 5, 3)]
    _both(ctx, monkeypatch, cells, method="redheffer", pe=1e-2)


def test_energy(ctx):
    a = ctx.order_powers([_pillar(11, 9, 7)], method="rcwa", nslices=6)[0]
    assert np.abs(a["R"].sum(1) + a["T"].sum(1) - 1.0).max() < 1e-10


@pytest.mark.parametrize("ends", [True, False])
@pytest.mark.parametrize("call", ["redheffer", "rcwa", "differential"])
@pytest.mark.parametrize("nx,ny", [(5, 3), (1, 9), (7, 7)])
def test_blocks(ctx, monkeypatch, call, ends, nx, ny):
    """Blocks in the full-order end modes: the same modes in the same order,
    the blocks to 1e-9 of their largest entry in the Fourier basis."""
    from tests.conftest import fourier_blocks
    ds = [_pillar(31, nx, ny, z1=0.12), _pillar(32, nx, ny, z1=0.15)]
    if not ends:
        for d in ds:
            d["end0"] = d["end1"] = None
    out = []
    for env in (None, "1"):
        monkeypatch.delenv("VRC_NO_FOLD", raising=False) if env is None else monkeypatch.setenv("VRC_NO_FOLD", env)
        out.append(ctx.redheffer(ds, pe=1e-2) if call == "redheffer" else getattr(ctx, call)(ds, 8))
    for a, b in zip(*out):
        for k in ("status", "n", "N", "n_eig", "n_samples", "n_nodes"):
            assert a[k] == b[k], k
        assert np.array_equal(a["gam0"], b["gam0"]) and np.array_equal(a["W1"], b["W1"])
        F, G = fourier_blocks(a), fourier_blocks(b)
        for k in F:
            assert np.abs(F[k] - G[k]).max() <= 1e-9 * max(np.abs(G[k]).max(), 1e-3), k


def _taper(nx=15):
    return st.taper_2d(norders=nx, length=0.6)


def _waveguide(spline):
    d = st.waveguide_pml(5, norders=5, ncontrol=4, length=0.4, spline=spline)
    w = 0.6 + 0.05 * d["widths"]
    d["xrules"] = [(i, zs, 2.0 + s * 0.5 * w) for (i, zs, _), s in zip(d["xrules"], (-1.0, 1.0))]
    return d


def _mesa():
    """Both axes moving, half-spaces, coordinates around the origin."""
    return dict(kind="grid", lam=1.1, nx=5, ny=7, pml=False, x=np.array([-0.5, -0.2, 0.2, 0.5]),
                y=np.array([-0.35, -0.1, 0.1, 0.35]),
                eps=np.array([[2.0, 2.0, 2.0], [2.0, 9.0 + 0.1j, 2.0], [2.0, 2.0, 2.0]], dtype=complex),
                xrules=[(1, [0.0, 0.2], [-0.2, -0.24]), (2, [0.0, 0.2], [0.2, 0.24])],
                yrules=[(1, [0.0, 0.2], [-0.1, -0.08]), (2, [0.0, 0.2], [0.1, 0.08])], z0=0.0, z1=0.2, end0=2.085,
                end1=1.0)


def _raster():
    rng = np.random.default_rng(3)
    q = rng.uniform(2.0, 8.0, (6, 5)) + 0j
    e = np.block([[q, q[:, ::-1]], [q[::-1], q[::-1, ::-1]]])
    return dict(kind="pixels", lam=1.0, nx=5, ny=5, pml=False, Lx=0.9, Ly=0.8, eps=e, z0=0.0, z1=0.2)


def _almost():
    """Symmetric at its ends and its middle only."""
    d = _mesa()
    d["xrules"] = [(1, [0.0, 0.05, 0.1, 0.2], [-0.2, -0.23, -0.2, -0.2]), (2, [0.0, 0.2], [0.2, 0.2])]
    return d


@pytest.mark.parametrize("make", [_taper, lambda: _waveguide(False), lambda: _waveguide(True), _mesa, _raster, _almost,
                                  lambda: st.planar_taper(w0=0.5, w1=0.6, length=0.6, norders=(7, 3))])
def test_tabulated_cells(ctx, monkeypatch, make):
    from tests.conftest import fourier_blocks
    d = make()
    out = []
    for env in (None, "1"):
        monkeypatch.delenv("VRC_NO_FOLD", raising=False) if env is None else monkeypatch.setenv("VRC_NO_FOLD", env)
        out.append((ctx.redheffer([d], pe=1e-2)[0], ctx.tree(0)))
    (a, ta), (b, tb) = out
    for k in ("status", "n", "N", "n_eig", "n_samples", "n_nodes"):
        assert a[k] == b[k], k
    assert [(x[0], x[1], x[3]) for x in ta] == [(x[0], x[1], x[3]) for x in tb]
    F, G = fourier_blocks(a), fourier_blocks(b)
    for k in F:
        assert np.linalg.norm(F[k] - G[k]) <= 1e-9 * max(np.linalg.norm(G[k]), 1e-3), k


def test_shifted_symmetry_takes_the_general_way(ctx, monkeypatch):
    """Symmetric about a point that is not the lattice origin: bit for bit the
    general way's result."""
    d = _mesa()
    d["x"] = d["x"] + 0.123
    d["xrules"] = [(i, zs, [v + 0.123 for v in vals]) for i, zs, vals in d["xrules"]]
    monkeypatch.delenv("VRC_NO_FOLD", raising=False)
    a = ctx.redheffer([d], pe=1e-2)[0]
    monkeypatch.setenv("VRC_NO_FOLD", "1")
    b = ctx.redheffer([d], pe=1e-2)[0]
    for k in ("Tdd", "Tuu", "Rud", "Rdu"):
        assert np.array_equal(a[k], b[k])


def _rim_pillar():
    """A pillar whose rim runs through pixel centres: by the rounding of
    x^2 + y^2 a centre lies inside and one of its mirror images outside.  Held
    to for every way a compiler may contract the raster's arithmetic."""
    from fractions import Fraction
    Lx, Ly, n = 0.41, 0.46, 59

    def fma(a, b, c):
        return float(Fraction(a) * Fraction(b) + Fraction(c))

    def coord(i, L, fused):
        h = L / n
        return fma(i + 0.5, h, -0.5 * L) if fused else (i + 0.5) * h - 0.5 * L

    def ranges(c, r):
        for fused in (False, True):
            d = {0: [], 1: [], 2: []}
            for i in (c, n - 1 - c):
                for j in (r, n - 1 - r):
                    x, y = coord(i, Lx, fused), coord(j, Ly, fused)
                    d[0].append(x * x + y * y)
                    d[1].append(fma(x, x, y * y))
                    d[2].append(fma(y, y, x * x))
            yield from ((min(v), max(v)) for v in d.values())

    for c in range(13, 22):
        for r in range(13, 22):
            lohi = list(ranges(c, r))
            lo, hi = max(a for a, _ in lohi), min(b for _, b in lohi)
            radius = np.sqrt(0.5 * (lo + hi))
            for _ in range(5):
                radius = np.nextafter(radius, 0.0)
            for _ in range(10):
                if lo <= radius * radius < hi:
                    radius = float(radius)
                    return _pillar(7, 5, 3, npx=n, npy=n, r0=radius, r1=radius, z1=0.2)
                radius = np.nextafter(radius, 1.0)
    raise AssertionError("no such radius")


def test_rim_pillar_is_asymmetric(ctx):
    d = _rim_pillar()
    P, Q = ctx.sample_pq(d, [0.1])
    m = d["nx"] * d["ny"]
    a, b = np.divmod(np.arange(m), d["ny"])
    worst = 0.0
    for perm in ((d["nx"] - 1 - a) * d["ny"] + b, a * d["ny"] + d["ny"] - 1 - b):
        q = np.concatenate([perm, m + perm])
        for M in (P[0], Q[0]):
            worst = max(worst, np.abs(np.abs(M[np.ix_(q, q)]) - np.abs(M)).max() / np.abs(M).max())
    assert worst > 1e-6


def _same_bits(a, b, keys):
    return all(np.array_equal(a[k], b[k]) for k in keys)


@pytest.mark.parametrize("max_depth", [1, 2])
@pytest.mark.parametrize("call", ["redheffer", "redheffer_forward", "order_powers"])
def test_late_asymmetry_with_a_capped_depth(ctx, monkeypatch, call, max_depth):
    """Found asymmetric below the root, in a tree that ends at its depth limit
    above the tolerance: bit for bit the general way's best effort."""
    out = []
    for env in (None, "1"):
        monkeypatch.delenv("VRC_NO_FOLD", raising=False) if env is None else monkeypatch.setenv("VRC_NO_FOLD", env)
        r = getattr(ctx, call)([_almost()], pe=1e-9, max_depth=max_depth)
        out.append(((r[0] if isinstance(r, tuple) else r)[0], ctx.tree(0)))
    (a, ta), (b, tb) = out
    assert a["status"] == b["status"] == 8
    assert _same_bits(a, b, ("R", "T") if call == "order_powers" else ("Tdd", "Tuu", "Rud", "Rdu", "W0", "W1"))
    assert ta == tb


@pytest.mark.parametrize("beside", [False, True])
@pytest.mark.parametrize("make", [_almost, _rim_pillar])
@pytest.mark.parametrize("call", ["order_powers", "blocks"])
@pytest.mark.parametrize("method", ["redheffer", "rcwa", "differential"])
def test_late_asymmetry(ctx, monkeypatch, method, call, make, beside):
    """Found asymmetric during the solve, alone and beside cells that are
    symmetric: bit for bit the general way's result."""
    cells = [make()]
    if beside:
        cells = [_mesa(), make(), _pillar(31, 5, 3, z1=0.12), make()]
    out = []
    for env in (None, "1"):
        monkeypatch.delenv("VRC_NO_FOLD", raising=False) if env is None else monkeypatch.setenv("VRC_NO_FOLD", env)
        if call == "order_powers":
            out.append(ctx.order_powers(cells, method=method, pe=1e-2, nslices=8))
        else:
            out.append(ctx.redheffer(cells, pe=1e-2) if method == "redheffer" else getattr(ctx, method)(cells, 8))
    for c in ((0,) if not beside else (1, 3)):
        a, b = out[0][c], out[1][c]
        assert a["status"] == b["status"] == 0
        assert _same_bits(a, b, ("R", "T") if call == "order_powers" else ("Tdd", "Tuu", "Rud", "Rdu", "W0", "W1"))
        if call == "blocks":
            assert all(a[k] == b[k] for k in ("N", "n_eig", "n_samples", "n_nodes"))


def test_first_pass_allocations(monkeypatch):
    """The classes' many small blocks come in no more pieces than the whole
    cells' few large ones, which take more memory."""
    from varrcwa_b200.capi import Context
    monkeypatch.setenv("VRC_LANES", "1")
    cells = [_pillar(40 + k, 7, 7, npx=32, npy=32) for k in range(300)]
    calls = []
    for env in (None, "1"):
        monkeypatch.delenv("VRC_NO_FOLD", raising=False) if env is None else monkeypatch.setenv("VRC_NO_FOLD", env)
        c = Context(0)
        before = c.kernel_stats()["host_alloc"]["bytes"]
        c.rcwa(cells, 4, blocks=False)
        calls.append(c.kernel_stats()["host_alloc"]["bytes"] - before)  # (of this entry: the number of calls)
        c.close()
    assert calls[0] <= calls[1]
