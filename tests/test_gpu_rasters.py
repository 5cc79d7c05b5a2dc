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


@pytest.mark.parametrize("nx,ny", [(t, 1) for t in range(35, 64, 2)] + [(1, 47)])
def test_toeplitz_every_wide_order(ctx, nx, ny):
    """Above 32 harmonics the shared memory that a launch asks for grows with each."""
    rng = np.random.default_rng(nx + 100 * ny)
    eps = rng.uniform(2.0, 12.0, (3, 5)) + 1j * rng.uniform(0.0, 0.5, (3, 5))
    d = dict(kind="pixels", lam=1.1, nx=nx, ny=ny, pml=False, Lx=0.9, Ly=0.7, eps=eps, z0=0.0, z1=0.4)
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


def _layers(nx, L, npix, seed, thick):
    rng = np.random.default_rng(seed)
    return dict(lam=0.9, Lx=0.7, Ly=0.7, nx=nx, ny=nx, layers=[rng.uniform(2.0, 4.0, (npix, npix)) for _ in range(L)],
                thick=[thick] * L, eps_in=1.0, eps_out=2.085)


def test_many_layers_in_groups(ctx):
    """Two stacks of 130 layers, whose pixel gradients come in two groups, bit
    for bit as each stack's alone, in one."""
    ds = [_layers(3, 130, 6, seed, 0.004) for seed in (1, 2)]
    w = np.zeros((2, 9))
    w[:, 4] = 1.0
    ctx.stack_forward(ds)
    g, gt = ctx.stack_backward(0.5 * w, w, want_thick=True)
    for k in range(2):
        ctx.stack_forward(ds[k:k + 1])
        g1, gt1 = ctx.stack_backward(0.5 * w[:1], w[:1], want_thick=True)
        assert np.abs(g1).max() > 0 and np.array_equal(g[k], g1[0]) and np.array_equal(gt[k], gt1[0])


def test_memory_of_many_layers():
    """What the backward pass of five stacks of 200 layers adds to the kept
    forward pass, in pool chunks: up to two of 64 MB for some 150 matrices of
    order 162, four of 27 MB for the block adjoints of a group of 255 layers, two
    of 64 MB for the groups' scratch and the gradients, and small ones; twelve of
    27 MB if the block adjoints of all 1000 layers were kept."""
    import torch
    from varrcwa_b200.capi import Context
    c = Context(0)
    try:
        w = np.zeros((5, 81))
        w[:, 40] = 1.0
        c.stack_forward([_layers(9, 200, 16, seed, 0.001) for seed in range(5)])
        before = torch.cuda.mem_get_info()[0]
        c.stack_backward(w, w)
        grown = before - torch.cuda.mem_get_info()[0]
    finally:
        c.close()
    assert grown < 400 << 20
