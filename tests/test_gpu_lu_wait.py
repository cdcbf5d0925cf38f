"""A wait of the LU panels that gives up: the call reports it, writes no result, and leaves the context fit for use.

The limit is set per context.  0 makes every block give up at the first column; with a few polls some blocks have
their columns in time and others do not, at other columns from run to run.
"""
import numpy as np
import pytest

import powerspectra_gpu as pg
from powerspectra_gpu import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 64, 400, 1100, 2100])
@pytest.mark.parametrize("limit", [0, 1, 2, 4])
def test_wait_gives_up(n, limit):
    ctx = pg.Context(0)
    rng = np.random.default_rng(n)
    M = np.asfortranarray(rng.normal(size=(n, n)) + 2.0 * n ** 0.5 * np.eye(n))
    b = rng.normal(size=(n, 2))
    want = ctx.solve(M, b)
    assert np.allclose(M @ want, b)
    for _ in range(5):
        ctx.check(ctx.lib.ps_lu_wait_limit(ctx.handle, limit))
        x = np.full((n, 2), 7.0, order="F")
        B = np.asfortranarray(b)
        st = ctx.lib.ps_solve(ctx.handle, _lib.dptr(M), n, n, _lib.dptr(B), 2, n, _lib.dptr(x), n)
        if limit == 0:
            assert st == _lib.PS_ERR_TIMEOUT
        if st:  # with some polls a wait may be long enough
            assert st == _lib.PS_ERR_TIMEOUT and np.all(x == 7.0)
        else:
            assert np.array_equal(x, want)
        ctx.check(ctx.lib.ps_lu_wait_limit(ctx.handle, 1 << 22))
        assert np.array_equal(ctx.solve(M, b), want)
    ctx.close()
