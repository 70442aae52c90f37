"""The eigen-solve at the edges of its kernels: one CTA / 8-CTA / 16-CTA cluster
tridiagonalisation, the two back-transformations, Jacobi above them."""
import numpy as np
import pytest

from gbhf import _lib

pytestmark = pytest.mark.gpu


def _check(ctx, a, tol=1.0):
    w, v = ctx.eigen_solve(a)
    wr = np.linalg.eigvalsh(a)
    sc = max(1.0, np.abs(wr).max())
    n = a.shape[0]
    assert np.all(np.diff(w) >= 0)
    np.testing.assert_allclose(w, wr, rtol=0, atol=1e-12 * sc)
    assert np.max(np.abs(a @ v - v * w)) < 1e-11 * sc
    assert np.max(np.abs(v.T @ v - np.eye(n))) < 1e-12


@pytest.mark.parametrize("n", [2, 15, 31, 33, 255, 256, 257, 304, 305, 607, 608, 609])
def test_sizes(ctx, n):
    a = np.random.default_rng(n).standard_normal((n, n))
    _check(ctx, a + a.T)


@pytest.mark.parametrize("n", [40, 240, 300, 520])
def test_repeated_and_clustered(ctx, n):
    """A third of the spectrum in exact multiplets, a third 1e-10 apart."""
    rng = np.random.default_rng(n)
    m = n // 3
    lam = np.concatenate([np.repeat(np.arange(1.0, 1.0 + (m + 3) // 4), 4)[:m], -5.0 + 1e-10 * np.arange(m),
                          np.linspace(20.0, 30.0, n - 2 * m)])
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    a = (q * lam) @ q.T
    _check(ctx, (a + a.T) / 2)


@pytest.mark.parametrize("n", [240, 320])
def test_diagonal_and_blocks(ctx, n):
    """No reflector has anything to do, and a matrix that falls apart into 2 x 2 blocks."""
    _check(ctx, np.diag(np.random.default_rng(n).permutation(n).astype(float)))
    _check(ctx, np.kron(np.diag(np.arange(1.0, n // 2 + 1)), [[2.0, 1.0], [1.0, 2.0]]))


def test_non_finite_matrix_is_reported(ctx):
    a = np.eye(300)
    a[7, 7] = np.nan
    with pytest.raises(_lib.NotConverged):
        ctx.eigen_solve(a)


@pytest.mark.parametrize("n", [2, 20, 200, 240, 300])
@pytest.mark.parametrize("power", [-520, -470, -401, 401, 500])
def test_elements_far_from_one(ctx, n, power):
    """A power of two on every element scales the eigenvalues by it and leaves the
    vectors as they are, also where squares of the elements leave the FP64 range."""
    a = np.random.default_rng(n).standard_normal((n, n))
    a = a + a.T
    w, v = ctx.eigen_solve(a * 2.0 ** power)
    w = w * 2.0 ** -power
    sc = max(1.0, np.abs(w).max())
    np.testing.assert_allclose(w, np.linalg.eigvalsh(a), rtol=0, atol=1e-12 * sc)
    assert np.max(np.abs(a @ v - v * w)) < 1e-11 * sc
    assert np.max(np.abs(v.T @ v - np.eye(n))) < 1e-12
