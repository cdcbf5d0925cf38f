"""The LU solve of the decoupling step (ps_lu.cu) at the edges of its panels, tiles and clusters.

Tolerance: Gaussian elimination with partial pivoting has a backward error of at most a few n eps growth
(growth below 10 for these matrices), so |M x - b| <= 1e-15 * 20 n (|M| |x| + |b|) per row bounds it with
room; the bar is that.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(M, b, x):
    n = M.shape[0]
    r = np.abs(M @ x - b)
    assert np.all(np.isfinite(x))
    assert np.all(r <= 2e-14 * n * (np.abs(M) @ np.abs(x) + np.abs(b)))


@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 63, 64, 65, 96, 127, 128, 129, 257, 500, 513, 1025, 2044, 4097])
@pytest.mark.parametrize("nrhs", [1, 3, 33])
def test_random_systems(ctx, n, nrhs):
    if n > 1100 and nrhs > 1:
        pytest.skip("the right-hand sides are covered at smaller n")
    rng = np.random.default_rng(n + nrhs)
    M = rng.normal(size=(n, n))  # needs its pivoting
    b = rng.normal(size=(n, nrhs))
    _check(M, b, ctx.solve(M, b))


@pytest.mark.parametrize("n", [5, 40, 97, 300])
def test_pivots_far_from_the_diagonal(ctx, n):
    rng = np.random.default_rng(n)
    P = np.eye(n)[rng.permutation(n)]
    b = rng.normal(size=n)
    np.testing.assert_array_equal(ctx.solve(P, b), P.T @ b)  # rows are only moved: exact
    M = np.tril(rng.normal(size=(n, n)))[::-1] + 1e-3 * rng.normal(size=(n, n))  # the largest entries last
    M[::-1][np.arange(n), np.arange(n)] += 4.0
    _check(M, b, ctx.solve(M, b))
    S = np.diag(2.0 ** rng.integers(-1030, 900, size=n).astype(float))[:, rng.permutation(n)]  # reciprocals overflow
    np.testing.assert_allclose(S @ ctx.solve(S, b * 1e-10), b * 1e-10, rtol=1e-13)


@pytest.mark.parametrize("n,zero", [(1, 0), (33, 32), (64, 5), (100, 99), (200, 0)])
def test_singular(ctx, n, zero):
    import powerspectra_gpu as pg
    M = np.eye(n) * 3.0
    M[zero] = 0.0
    with pytest.raises(pg.PowerSpectraArgumentError, match=r"singular \(zero pivot %d\)" % (zero + 1)):
        ctx.solve(M, np.ones(n))
    assert np.allclose(ctx.solve(np.eye(n) * 2, np.ones(n)), 0.5)
