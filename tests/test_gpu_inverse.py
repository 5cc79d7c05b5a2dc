"""The blocked inversion at the edges of its panels (16 columns up to n = 512, 8
above, one or two rows per thread) against the identity, and matrices whose
pivots lie far from the diagonal.  Residual bound: eps n cond, with room of 50."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from varrcwa_b200.capi import Context
    c = Context(0)
    yield c
    c.close()


def _check(ctx, A):
    X, st = ctx.zinv(A)
    n = A.shape[-1]
    assert not np.any(st)
    for b in range(A.shape[0]):
        bound = 50 * 2.2e-16 * n * np.linalg.cond(A[b])
        assert np.abs(A[b] @ X[b] - np.eye(n)).max() < bound


@pytest.mark.parametrize("n", [31, 32, 33, 47, 48, 49, 64, 65, 255, 256, 257, 272, 511, 512, 513, 520, 527])
def test_orders(ctx, n):
    rng = np.random.default_rng(n)
    _check(ctx, rng.standard_normal((2, n, n)) + 1j * rng.standard_normal((2, n, n)))


@pytest.mark.parametrize("n", [2, 3, 7, 8, 9, 30, 63, 66, 95, 96, 97])
def test_small_orders(ctx, n):
    """The registers' edges, more matrices than one wave takes."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((300, n, n)) + 1j * rng.standard_normal((300, n, n))
    A[:, np.arange(n), np.arange(n)] += 2.0 * n
    _check(ctx, A)


@pytest.mark.parametrize("n", [2, 20, 63, 90])
def test_small_pivots(ctx, n):
    """Pivots far from the diagonal and far from one; singular, infinite and
    undefined entries are reported for their own matrix alone."""
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    P = np.eye(n)[::-1] * rng.uniform(0.5, 2.0, n)[:, None] + 0j
    for A in (P, P + 1e-3 * G, 1e-160 * G, 1e160 * G):
        X, st = ctx.zinv(A)
        bound = 50 * 2.2e-16 * n * np.linalg.cond(A / np.abs(A).max())
        assert st == 0 and np.abs(A @ X - np.eye(n)).max() < bound
    A = np.stack([G] * 5)
    A[1, :, 0] = 0.0
    A[2, 1, 0] = np.inf
    A[3, :, 0] = np.nan
    assert list(ctx.zinv(A)[1]) == [0, 4, 4, 4, 0]


@pytest.mark.parametrize("n", [1025, 1056, 2049, 2767])
def test_beyond_structures(ctx, n):
    """Orders that no structure has (six rows per thread, 4 columns): rows of a
    diagonal in [1, 2] exchanged, and 0.1 / sqrt(n) of noise, whose 2-norm stays
    below 0.3, so cond < 2.3 / 0.7 < 4.  The next order is refused."""
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) * (0.1 / np.sqrt(n))
    A[np.arange(n), np.arange(n)] += rng.uniform(1.0, 2.0, n)
    A = A[rng.permutation(n)]
    X, st = ctx.zinv(A)
    assert st == 0 and np.abs(A @ X - np.eye(n)).max() < 50 * 2.2e-16 * n * 4
    with pytest.raises(Exception):
        ctx.zinv(np.eye(2768, dtype=complex))


@pytest.mark.parametrize("n", [40, 70, 300, 530])
def test_far_pivots(ctx, n):
    """A scaled permutation (every pivot off the diagonal), and rows of very
    different size."""
    rng = np.random.default_rng(n)
    P = np.eye(n)[rng.permutation(n)] * rng.uniform(0.5, 2.0, n)[:, None] + 0j
    G = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    _check(ctx, np.stack([P, P + 1e-3 * G, G * 10.0 ** rng.uniform(-3, 3, n)[:, None]]))


@pytest.mark.parametrize("n", [40, 300, 530])
def test_singular(ctx, n):
    A = np.ones((2, n, n), dtype=complex)
    A[1] = np.eye(n)
    A[1, 5, 5] = 0.0
    assert list(ctx.zinv(A)[1]) == [4, 4]


@pytest.mark.parametrize("n", [97, 130, 300, 530])
def test_undefined_entries(ctx, n):
    """Panels: infinite and undefined entries are reported for their own matrix
    alone, wherever the entry's panel is."""
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A = np.stack([G] * 7)
    A[1, 1, 0] = np.inf
    A[2, 5, n - 1] = np.nan
    A[3, :, n // 2] = np.nan
    A[4, n - 1, n // 2] = complex(0.0, np.inf)
    A[5, :, n - 2] = 0.0
    assert list(ctx.zinv(A)[1]) == [0, 4, 4, 4, 4, 4, 0]
