"""The plain FP64 kernel's forms (windows per class) at the edges of its 32-point refills and tiles.

Tolerance: 1e-12 of the sum of |terms| behind each element, the bar of every plain FP64 test: the
oracle's recurrences and the kernel's each carry rounding errors that grow no faster than the family
length (below 2e-14 relative at these sizes), so the bar leaves a factor of 50.
"""
import numpy as np
import pytest

from gpu_util import cond_scale, max_err_scaled
from oracle import oracle as o

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def _W(nW, seed):
    from powerspectra_gpu import synthetic as syn
    return syn.mask_spectrum(nW, 0.6, max(nW / 3.0, 5.0), seed=seed)


@pytest.mark.parametrize("L,lmin", [(0, 0), (1, 0), (2, 0), (3, 2), (30, 0), (31, 0), (32, 0), (33, 1), (62, 0), (63, 0),
                                    (64, 0), (65, 2), (95, 0), (96, 0), (127, 3)])
def test_every_case_mask(ctx, L, lmin):
    Ws = {s: _W(2 * L + 1, s + 3) for s in range(4)}
    ref = {s: o.inner_mcm(s, Ws[s], lmin, L) for s in range(4)}
    scale = {s: cond_scale(s, Ws[s], lmin, L) for s in range(4)}
    for cases in range(1, 16):
        sel = {s: Ws[s] for s in range(4) if cases >> s & 1}
        got = ctx.mcm_multi(sel, lmin, L)
        for s in sel:
            assert max_err_scaled(got[s], ref[s], scale[s]) < RTOL, (cases, s)


@pytest.mark.parametrize("L,lmin,K", [(33, 0, 1), (64, 2, 3), (65, 0, 5), (96, 0, 8)])
def test_xi_every_product_and_parity(ctx, L, lmin, K):
    Ws = [_W(2 * L + 1, 20 + k) for k in range(K)]
    for product in range(3):
        for parity in range(3):
            got = ctx.xi(product, parity, Ws, lmin, L)
            for k in range(K):
                ref = o.xi(product, parity, Ws[k], lmin, L)
                scale = np.abs(ref)
                if product == 2:  # terms of both signs: the Cauchy-Schwarz bound on their sum
                    scale = np.sqrt(np.abs(o.xi(0, 0, Ws[k], lmin, L) * o.xi(1, 0, Ws[k], lmin, L)))
                assert max_err_scaled(got[k], ref, scale) < RTOL, (product, parity, k)


@pytest.mark.parametrize("K,cases,slots", [(4, 0x5, None), (4, 0xF, None), (3, 0x7, None),
                                           (8, 0xC, {(k, 2) for k in range(7)} | {(0, 3)}),
                                           (8, 0xC, {(k, 3) for k in range(8)}), (7, 0x2, None)])
def test_set_groups(ctx, K, cases, slots):
    L = 65
    Ws = [_W(2 * L + 1, 40 + k) for k in range(K)]
    got = ctx.mcm_set(cases, Ws, 1, L, mode="plain", slots=slots)
    for (k, s), M in got.items():
        assert max_err_scaled(M, o.inner_mcm(s, Ws[k], 1, L), cond_scale(s, Ws[k], 1, L)) < RTOL, (k, s)
