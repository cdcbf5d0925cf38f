"""The 2 x 2 block matrices written whole, against the ++ and -- matrices of the same pass, and results in new and
in strided host memory: equal numbers."""
import numpy as np
import pytest

import powerspectra_gpu as pg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,lmin", [(0, 0), (1, 1), (31, 0), (32, 0), (65, 2), (200, 200), (257, 3)])
@pytest.mark.parametrize("mode", ["plain", "chosen"])
def test_blocks_equal_their_parts(ctx, L, lmin, mode):
    from powerspectra_gpu import synthetic as syn
    W = syn.mask_spectrum(2 * L + 1, 0.5, max(L / 2.0, 5.0), seed=9)
    part = ctx.mcm_multi({2: W, 3: W}, lmin, L, mode=mode)
    pp, mm = part[2], part[3]
    want = np.block([[pp, mm], [mm, pp]]), np.block([[pp, -mm], [-mm, pp]])
    for ask in ((True, False), (False, True), (True, True)):
        got = ctx.mcm_blocks(W, lmin, L, mode=mode, ee_bb=ask[0], eb_be=ask[1])
        for g, w, a in zip(got, want, ask):
            assert (g is None) if not a else (g.flags.f_contiguous and np.array_equal(g, w))
            if a:
                assert np.array_equal(np.signbit(g), np.signbit(w))


def test_blocks_refuse_what_the_parts_refuse(ctx):
    W = np.ones(9)
    for lmin, lmax in ((5, 4), (9, 4), (-1, 4)):
        with pytest.raises(pg.PowerSpectraArgumentError):
            ctx.mcm_blocks(W, lmin, lmax)
    with pytest.raises(pg.PowerSpectraArgumentError):
        ctx.mcm_blocks(W, 0, 4, ee_bb=False)
    for spec in ("EE_BB", "EB_BE", ("EE_BB", "EB_BE")):
        with pytest.raises(pg.PowerSpectraArgumentError):
            pg.mcm(spec, W, lmin=9, lmax=4, ctx=ctx)


@pytest.mark.parametrize("gap", [0, 3, 20000])  # the pages of the whole range, and column by column
def test_results_in_new_and_strided_memory(ctx, gap):
    from powerspectra_gpu import _lib, synthetic as syn
    L = 399  # 1.28 MB
    n, ld = L + 1, L + 1 + gap
    W = syn.mask_spectrum(n, 0.5, 100.0, seed=4)
    want = ctx.mcm(0, W, 0, L)
    for filled in (False, True):
        M = np.zeros((n, ld))  # rows here are columns of the column-major result
        if filled:
            M[:] = 7.0
        ctx.check(ctx.lib.ps_mcm(ctx.handle, 0, _lib.dptr(W), n, 0, L, _lib.mode_code("plain"), _lib.dptr(M), ld))
        assert np.array_equal(M[:, :n].T, want)
        assert bool((M[:, n:] == (7.0 if filled else 0.0)).all())
