"""ps_launch_count counts the kernels of a solve: per panel of 32 columns the panel itself, the rows and the product of
the next panel's columns and of all others, and one kernel per 32 rows of the back substitution.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,want", [(1, 1 + 1 + 1), (32, 1 + 1 + 1), (64, (1 + 2 + 2) + (1 + 1) + 2),
                                    (96, (1 + 2 + 2) + (1 + 2 + 2) + (1 + 1) + 3)])
def test_count(ctx, n, want):
    ctx.solve(2.0 * np.eye(n), np.ones(n))
    before = ctx.launch_count()
    ctx.solve(2.0 * np.eye(n), np.ones(n))
    assert ctx.launch_count() - before == want
