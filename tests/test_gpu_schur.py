"""The eigensolver at the edges of its QR kernel: window and strip remainders,
the smallest orders, the order from which deflation windows run, and entries
whose squares leave the double range.  Residuals against numpy in FP64, with
the bound of the other eigensolver tests (1e-12 n of the matrix's scale)."""
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
    lam, W = ctx.eig(A)
    n = A.shape[-1]
    for b in range(A.shape[0]):
        scale = np.abs(A[b]).max()
        assert np.abs(A[b] @ W[b] - W[b] * lam[b][None, :]).max() <= 1e-12 * scale * n
        assert np.abs(np.linalg.norm(W[b], axis=0) - 1.0).max() < 1e-12


@pytest.mark.parametrize("n", [2, 3, 4, 5, 11, 12, 13, 31, 32, 33, 55, 56, 57, 58, 59, 61, 64, 97, 127, 128, 129, 131,
                               165])
def test_orders(ctx, n):
    rng = np.random.default_rng(n)
    _check(ctx, rng.standard_normal((3, n, n)) + 1j * rng.standard_normal((3, n, n)))


@pytest.mark.parametrize("n", [2, 3, 8, 9, 32, 33, 48, 49, 64, 65, 80, 81, 95, 96, 97, 111, 112, 113, 114])
def test_reduced_columns(ctx, n):
    """Reflectors at the edges of the small reduction's lanes and columns,
    with columns that need none."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((4, n, n)) + 1j * rng.standard_normal((4, n, n))
    A[1] = np.triu(A[1], -1)
    A[2, 2:, : n // 2] = 0
    A[3] = np.diag(np.diagonal(A[3]))
    _check(ctx, A)


@pytest.mark.parametrize("n,batch", [(114, 1), (127, 150), (160, 2), (192, 1), (193, 1), (256, 1), (257, 1), (513, 1)])
def test_panels(ctx, n, batch):
    """Row slots and column groups of the reduction's panels."""
    rng = np.random.default_rng(n)
    _check(ctx, rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n)))


@pytest.mark.parametrize("n", [159, 160, 230])
def test_teams(ctx, n):
    """However many CTAs a matrix gets, the eigenvalues are the same bits."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((1, n, n)) + 1j * rng.standard_normal((1, n, n))
    _check(ctx, A)
    one = ctx.eig(A)[0][0]
    for batch in (9, 10, 29, 30, 37, 38):
        lam = ctx.eig(np.repeat(A, batch, axis=0))[0]
        assert all(np.array_equal(x, one) for x in lam)


@pytest.mark.parametrize("scale", [1e-120, 1e-75, 1e60])
@pytest.mark.parametrize("n", [13, 140])
def test_scaled(ctx, n, scale):
    rng = np.random.default_rng(n)
    _check(ctx, scale * (rng.standard_normal((2, n, n)) + 1j * rng.standard_normal((2, n, n))))


@pytest.mark.parametrize("n", [30, 150])
def test_structured(ctx, n):
    """Graded rows, a diagonal matrix, exact zeros on the subdiagonal, a
    cyclic shift (all eigenvalues of modulus one)."""
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    graded = G * 10.0 ** (-8.0 * np.arange(n) / n)[:, None]
    diag = np.diag(np.arange(n) + 1.0).astype(complex)
    block = np.triu(G)
    block[: n // 2, : n // 2] += np.tril(G[: n // 2, : n // 2], -1)
    shift = np.roll(np.eye(n), 1, axis=0).astype(complex)
    _check(ctx, np.stack([graded, diag, block, shift]))


@pytest.mark.parametrize("n", [2, 18, 70, 150])
def test_equal_diagonals(ctx, n):
    """Multiple eigenvalues up to rounding: the modes of a uniform medium, and
    blocks with equal diagonal entries whose off-diagonal product is below
    their rounding."""
    rng = np.random.default_rng(n)
    d = -2e4 * np.repeat(rng.uniform(0.1, 1.0, n // 2), 2)
    A = np.tile(np.diag(d).astype(complex), (12, 1, 1))
    A[:8] += 2e-12 * rng.standard_normal((8, n, n))
    i = np.arange(0, n, 2)
    A[8:, i, i + 1] = -1.85e-12 * 10.0 ** rng.uniform(-1, 1, (4, n // 2))
    A[8:, i + 1, i] = -1.05e-13 * 10.0 ** rng.uniform(-1, 1, (4, n // 2))
    _check(ctx, A)


@pytest.mark.parametrize("n", [114, 115, 116])
def test_reduction_at_the_end_of_shared_memory(ctx, monkeypatch, n):
    """The reduction in shared memory takes every order whose matrix has room
    there, (n + 10) n + 8 entries: bit for bit VRC_HESS_BLOCKED=0 up to it and
    VRC_HESS_BLOCKED=1 above."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((4, n, n)) + 1j * rng.standard_normal((4, n, n))
    A[1] = np.triu(A[1], -1)
    A[2, 2:, : n // 2] = 0
    A[3] = np.diag(np.diagonal(A[3]))
    monkeypatch.delenv("VRC_HESS_BLOCKED", raising=False)
    _check(ctx, A)
    W = ctx.eig(A)[1]
    monkeypatch.setenv("VRC_HESS_BLOCKED", "0" if 16 * ((n + 10) * n + 8) <= 227 * 1024 else "1")
    assert np.array_equal(ctx.eig(A)[1], W)
