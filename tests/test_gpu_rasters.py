"""The raster stages at the edges of their tiles, against the oracle: P and Q
(1e-12 relative, as the other assembly tests) and the pixel gradients of a
stack (1e-9 of the largest, as the small stack of the adjoint tests), with
rectangular rasters and unequal harmonic counts; and the differential method's
slices for a batch of unequal slices (1e-9, as the integrators' tests)."""
import numpy as np
import pytest

from oracle import varrcwa_oracle as O
from oracle.stack_adjoint import Stack, stack_backward, stack_forward
from oracle.structures_adapter import end_bases, make_sampler
from tests.cases import CASES
from tests.conftest import fourier_blocks, relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npy,npx", [(1, 1), (1, 17), (15, 16), (16, 64), (65, 33), (31, 129)])
@pytest.mark.parametrize("nx,ny", [(1, 3), (9, 1), (5, 7)])
def test_pq(ctx, npy, npx, nx, ny):
    rng = np.random.default_rng(npy * npx)
    eps = rng.uniform(2.0, 12.0, (npy, npx)) + 1j * rng.uniform(0.0, 0.5, (npy, npx))
    d = dict(kind="pixels", lam=1.1, nx=nx, ny=ny, pml=False, Lx=0.9, Ly=0.7, eps=eps, z0=0.0, z1=0.4)
    P, Q = ctx.sample_pq(d, [0.1, 0.2, 0.3])
    oP, oQ = make_sampler(d).sample(0.1)
    for k in range(3):
        assert relerr(P[k], oP) < 1e-12 and relerr(Q[k], oQ) < 1e-12


@pytest.mark.parametrize("npy,npx,nx,ny", [(33, 70, 3, 5), (64, 17, 9, 1)])
def test_many_samples(ctx, npy, npx, nx, ny):
    """The Fourier products of many samples at once, bit for bit those of one."""
    rng = np.random.default_rng(npx)
    eps = rng.uniform(2.0, 12.0, (npy, npx)) + 1j * rng.uniform(0.0, 0.5, (npy, npx))
    d = dict(kind="pixels", lam=1.1, nx=nx, ny=ny, pml=False, Lx=0.9, Ly=0.7, eps=eps, z0=0.0, z1=0.4)
    P, Q = ctx.sample_pq(d, [0.1])
    Pm, Qm = ctx.sample_pq(d, np.linspace(0.0, 0.4, 160))
    assert all(np.array_equal(x, P[0]) for x in Pm) and all(np.array_equal(x, Q[0]) for x in Qm)


@pytest.mark.parametrize("nx,ny", [(7, 9), (11, 3), (1, 13), (15, 1), (1, 17), (23, 1), (1, 25), (31, 1), (33, 1), (1, 41),
                                   (63, 1)])
def test_toeplitz_orders(ctx, nx, ny):
    """The Toeplitz inverses at the edges of their widths."""
    rng = np.random.default_rng(nx + ny)
    eps = rng.uniform(2.0, 12.0, (2, 5, 7)) + 1j * rng.uniform(0.0, 0.5, (2, 5, 7))
    for e in eps:
        d = dict(kind="pixels", lam=1.1, nx=nx, ny=ny, pml=False, Lx=0.9, Ly=0.7, eps=e, z0=0.0, z1=0.4)
        P, Q = ctx.sample_pq(d, [0.1])
        oP, oQ = make_sampler(d).sample(0.1)
        assert relerr(P[0], oP) < 1e-12 and relerr(Q[0], oQ) < 1e-12


@pytest.mark.parametrize("npy,npx,nx,ny", [(7, 12, 3, 3), (12, 7, 3, 5), (9, 33, 5, 1), (16, 8, 1, 5), (10, 17, 5, 3)])
def test_pixel_gradients(ctx, npy, npx, nx, ny):
    rng = np.random.default_rng(npx)
    L, C = 3, 2
    stacks = [dict(lam=0.633, Lx=0.6, Ly=0.5, nx=nx, ny=ny, layers=[rng.uniform(2.0, 6.0, (npy, npx)) for _ in range(L)],
                   thick=list(rng.uniform(0.1, 0.2, L)), eps_in=1.0, eps_out=2.085) for _ in range(C)]
    w = rng.uniform(0.0, 1.0, (2, C, nx * ny))
    ctx.stack_forward(stacks)
    g, gt = ctx.stack_backward(w[0], w[1], want_thick=True)
    for c, d in enumerate(stacks):
        st = Stack(d["lam"], nx, ny, d["Lx"], d["Ly"], d["layers"], d["thick"], d["eps_in"], d["eps_out"])
        tp = stack_forward(st)[2]
        og, ogt = stack_backward(st, tp, w[0, c], w[1, c], want_thick=True)
        assert np.abs(g[c] - np.array(og)).max() <= 1e-9 * np.abs(og).max()
        assert np.abs(gt[c] - np.array(ogt)).max() <= 1e-9 * np.abs(ogt).max()


def test_differential_batch_of_unequal_slices(ctx):
    base = CASES["asym_diff"]["desc"]
    ds = [dict(base, lam=base["lam"] * f, z1=base["z1"] * f) for f in (0.2, 0.25)]
    for d, r in zip(ds, ctx.differential(ds, 5)):
        s = make_sampler(d)
        e0, e1 = end_bases(d, s)
        G = O.differential_compute(s, d["z0"], d["z1"], 5, e0, e1).fourier_blocks()
        F = fourier_blocks(r)
        for k in F:
            assert relerr(F[k], G[k]) < 1e-9, k
