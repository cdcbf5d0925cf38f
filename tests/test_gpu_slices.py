"""The table of window slices of the chosen kernels: slices that begin below l3 = 0 or end beyond 2 lmax at
small sizes and lmin > 0, and a batch whose tables do not all fit.

Tolerance: 1e-6 of the sum of |terms| behind each element, the bar of the chosen mode (FP32 products against
FP64).  A slice is the same whether it comes from a table or not, so equal problems give equal bits.
"""
import numpy as np
import pytest

from gpu_util import cond_scale, max_err_scaled
from oracle import oracle as o

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

RTOL = 1e-6


def _W(nW, seed):
    from powerspectra_gpu import synthetic as syn
    return syn.mask_spectrum(nW, 0.5, max(nW / 3.0, 5.0), seed=seed)


@pytest.mark.parametrize("L,lmin", [(0, 0), (1, 1), (2, 0), (30, 29), (31, 0), (32, 1), (33, 33), (63, 31), (64, 0), (97, 60), (128, 0), (129, 70)])
@pytest.mark.parametrize("full", [True, False])
def test_slices_at_the_ends(ctx, L, lmin, full):
    nW = 2 * L + 1 if full else L // 2 + 1  # with windows that end early too
    Ws = {s: _W(nW, 50 + s) for s in range(4)}
    for sel in ((0,), (1,), (2,), (3,), (2, 3), (0, 1, 2, 3)):
        got = ctx.mcm_multi({s: Ws[s] for s in sel}, lmin, L, mode="chosen")
        for s in sel:
            full_W = np.concatenate([Ws[s], np.zeros(2 * L + 1 - nW)])
            ref, scale = o.inner_mcm(s, full_W, lmin, L), cond_scale(s, full_W, lmin, L)
            assert max_err_scaled(got[s], ref, scale) < RTOL, (sel, s)


@pytest.mark.parametrize("L,lmin", [(0, 0), (31, 0), (33, 2), (64, 1), (127, 0), (128, 0)])
def test_sets(ctx, L, lmin):
    Ws = [_W(2 * L + 1, 70 + k) for k in range(3)]
    got = ctx.mcm_set(0xF, Ws, lmin, L, mode="chosen")
    for (k, s), M in got.items():
        assert max_err_scaled(M, o.inner_mcm(s, Ws[k], lmin, L), cond_scale(s, Ws[k], lmin, L)) < RTOL, (k, s)


def test_batch_beyond_the_tables(ctx):
    """Groups of lmax 128 and more have a table, 603 kB each here; the last of them have no room for it."""
    sizes, K, n = [128, 127, 160, 128, 128, 130, 128, 128], 1, 4800
    Ws = [[_W(2 * L + 1, 10 * i + k) for k in range(K)] for i, L in enumerate(sizes)]
    dW = [[torch.tensor(w, device="cuda") for w in set_] for set_ in Ws]
    dM = [torch.zeros((n // 8, K, L + 1, L + 1), dtype=torch.float64, device="cuda") for L in sizes]
    probs = [{"lmin": 0, "lmax": sizes[i % 8], "cases": 0x1, "nW": 2 * sizes[i % 8] + 1, "ldm": sizes[i % 8] + 1,
              "W": [w.data_ptr() for w in dW[i % 8]],
              "M": [p for k in range(K) for p in (dM[i % 8][i // 8, k].data_ptr(), 0, 0, 0)]} for i in range(n)]
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    try:
        ctx.batch_prepare(probs, group_slots=8)
        for run in (ctx.batch_run, ctx.batch_graph_launch):
            for m in dM:
                m.zero_()
            torch.cuda.synchronize()
            run()
            torch.cuda.synchronize()
            for i, L in enumerate(sizes):
                assert bool((dM[i] == dM[i][0]).all())
                for k in range(K):
                    ref, scale = o.inner_mcm(0, Ws[i][k], 0, L), cond_scale(0, Ws[i][k], 0, L)
                    assert max_err_scaled(dM[i][0, k].cpu().numpy().T, ref, scale) < RTOL, (i, k)
    finally:
        ctx.set_stream(0)
