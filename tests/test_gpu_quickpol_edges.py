"""The plain QuickPol kernel at the smallest grids and bands, and where equal spins run one family.

Tolerance: 1e-12 of the sum of |W f1 f2| behind each element, as for every plain QuickPol test.  The
recurrences' rounding grows with the family length (below 2e-14 at these sizes) and with how far the
spins reach into the classically forbidden ends (a factor of 10 at most for these).
"""
import numpy as np
import pytest

from oracle import oracle as o

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu1,nu2,s1,s2", [(0, 0, 0, 0), (0, 0, 2, 2), (3, 3, -1, -1), (2, 2, -2, -2), (5, 5, 0, 0),
                                           (0, 0, 2, -2), (1, 0, 1, 2), (0, 6, 0, 1), (-2, 2, 2, 2)])
@pytest.mark.parametrize("lmax,bl,bu", [(2, 0, 0), (3, 1, 0), (5, 9, 9), (8, 0, 3), (33, 2, 40), (65, 7, 7)])
def test_small_grids(ctx, nu1, nu2, s1, s2, lmax, bl, bu):
    rng = np.random.default_rng(lmax)
    for nW in (2 * lmax + 1, lmax):
        W = rng.normal(size=nW)
        R = o.quickpol_xi(nu1, nu2, s1, s2, W, lmax, bl, bu, common_match=True)
        scale = o.quickpol_xi(nu1, nu2, s1, s2, W, lmax, bl, bu, absolute=True)
        G = ctx.quickpol_xi(nu1, nu2, s1, s2, W, lmax, bl, bu)
        assert np.all(np.isfinite(G))
        assert not np.any(G[scale == 0])
        assert np.max(np.abs(G - R)[scale > 0] / scale[scale > 0], initial=0.0) < 1e-12


def test_equal_spins_chosen_same_bits(ctx):
    """The one-family form of the chosen kernel against its two-family form with the spins of one family
    negated: (l' l l''; m) and (l' l l''; -m) differ by a sign that is the same for all l' of one parity
    of l + l' + l'', so on a spectrum of even entries alone the sums agree up to that sign."""
    lmax, b = 90, 12
    W = np.zeros(2 * lmax + 1)
    W[::2] = np.random.default_rng(1).random(lmax + 1)
    A = ctx.quickpol_xi(0, 0, 2, 2, W, lmax, b, b, mode="chosen")
    B = ctx.quickpol_xi(0, 0, 2, -2, W, lmax, b, b, mode="chosen")
    scale = o.quickpol_xi(0, 0, 2, 2, W, lmax, b, b, absolute=True)
    assert np.max(np.abs(np.abs(A) - np.abs(B))[scale > 0] / scale[scale > 0]) < 1e-6
