"""Mask spectra of more terms than the reduction takes at a time, at lout that are no multiple of its 32 columns.

Tolerance: 1e-14 of the mean of sum |a| |b| per l.  A term's sum has at most 2 lmax + 1 = 1201 products in chains of a
few dozen, and at most 16 terms are added: some 60 roundings of 1.1e-16 in a row, 7e-15 at the worst.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nterms", [4, 5, 8, 9, 16])
@pytest.mark.parametrize("lmax,mmax,lout", [(600, 600, 600), (600, 333, 577), (95, 95, 33), (40, 7, 31), (0, 0, 0)])
def test_terms(ctx, nterms, lmax, mmax, lout):
    rng = np.random.default_rng(nterms + lmax)
    nalm = (mmax + 1) * (mmax + 2) // 2 + (mmax + 1) * (lmax - mmax)
    sets = [rng.normal(size=nalm) + 1j * rng.normal(size=nalm) for _ in range(nterms + 1)]
    A, B = sets[:nterms], sets[1:]
    B[0] = A[0]  # an auto-spectrum
    A[-1] = None if nterms == 9 else A[-1]  # an all-zero set still counts
    ref, scale = np.zeros(lout + 1), np.zeros(lout + 1)
    for l in range(lout + 1):
        m = np.arange(min(l, mmax) + 1)
        at = m * (2 * lmax + 1 - m) // 2 + l
        w = np.where(m == 0, 1.0, 2.0)
        for a, b in zip(A, B):
            if a is not None:
                ref[l] += np.sum(w * (a[at] * np.conj(b[at])).real) / (2 * l + 1)
                scale[l] += np.sum(w * np.abs(a[at]) * np.abs(b[at])) / (2 * l + 1)
    got = ctx.window_W(A, B, lmax, mmax=mmax, lout=lout)
    assert np.all(np.abs(got - ref / nterms) <= 1e-14 * scale / nterms)
