"""The LU solve where a panel has more than 128 rows per block (n above 2048) and with as many right-hand sides as it
takes.  The bar is that of the smaller systems: a backward error of at most 2e-14 n of |M| |x| + |b| per row.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nrhs", [(40, 32), (1000, 32), (1024, 31), (2049, 1), (2049, 32), (3000, 7), (4095, 1), (4096, 32)])
def test_large_panels(ctx, n, nrhs):
    rng = np.random.default_rng(n + nrhs)
    M = rng.normal(size=(n, n))  # needs its pivoting
    b = rng.normal(size=(n, nrhs))
    x = ctx.solve(M, b)
    assert np.all(np.isfinite(x))
    assert np.all(np.abs(M @ x - b) <= 2e-14 * n * (np.abs(M) @ np.abs(x) + np.abs(b)))
