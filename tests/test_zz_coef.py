"""The chosen kernels with and without the table of square-root ratios: the same numbers, so the same bits.

The context has a table from lmax 512 on, the allocation-free entry point none.  A larger table, left by a call
of larger lmax, holds the same rows.  A batch has a table at every lmax.
"""
import ctypes

import numpy as np
import pytest

from test_zz_no_alloc import _noalloc_fn

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _windows(nW):
    from powerspectra_gpu import synthetic as syn
    return [torch.tensor(syn.mask_spectrum(nW, 0.4 + 0.1 * s, nW / 4.0, seed=60 + s), device="cuda") for s in range(4)]


def _both(ctx, cases, lmin, lmax):
    fn, L = _noalloc_fn()
    used, n, nW = [s for s in range(4) if cases >> s & 1], lmax - lmin + 1, 2 * lmax + 1
    dW = _windows(nW)
    new, ref = ({s: torch.zeros((n, n), dtype=torch.float64, device="cuda") for s in used} for _ in range(2))
    ptr = lambda d: L.dptr_array([d[s].data_ptr() if s in d else 0 for s in range(4)])
    assert fn(cases, L.dptr_array([d.data_ptr() for d in dW]), nW, lmin, lmax, ptr(ref), n,
              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    ctx.mcm_multi_device({s: dW[s].data_ptr() for s in used}, nW, lmin, lmax, {s: new[s].data_ptr() for s in used}, n,
                         mode="chosen")
    torch.cuda.synchronize()
    return new, ref


@pytest.mark.parametrize("lmax,lmin", [(511, 0), (512, 0), (543, 30), (544, 2), (800, 0), (513, 500), (512, 512)])
def test_table_and_no_table(lmax, lmin):
    from powerspectra_gpu import Context
    ctx = Context(0)  # its own: the table starts at this size
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    for again in (False, True):
        if again:  # a larger table, read by the smaller calls
            _both(ctx, 0xF, lmin, lmax + 37)
        for cases in (0xF, 0xC, 0x4, 0x8):
            new, ref = _both(ctx, cases, lmin, lmax)
            for s in new:
                assert bool((new[s] == ref[s]).all()), (cases, s, again)


@pytest.mark.parametrize("sizes", [(1, 33, 64), (95, 700, 31)])
def test_batch_with_a_table(sizes):
    from powerspectra_gpu import Context
    ctx = Context(0)
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    want, probs, keep = [], [], []
    for lmax in sizes:
        for cases in (0xF, 0xC):
            new, ref = _both(ctx, cases, 0, lmax)
            dW, n = _windows(2 * lmax + 1), lmax + 1
            M = {s: torch.zeros((n, n), dtype=torch.float64, device="cuda") for s in ref}
            keep.append((dW, M))
            want.append(ref)
            spins = [s for s in range(4) if cases >> s & 1]
            W = dW[spins[0]]  # a problem has one window for its cases: compare those of the window's own case
            probs.append({"lmin": 0, "lmax": lmax, "cases": cases, "nW": 2 * lmax + 1, "ldm": n, "W": [W.data_ptr()],
                          "M": [M[s].data_ptr() if s in M else 0 for s in range(4)]})
    ctx.batch_prepare(probs, group_slots=4)
    ctx.batch_run()
    torch.cuda.synchronize()
    for (dW, M), ref in zip(keep, want):
        s = min(ref)
        d = (M[s] - ref[s]).abs().max().item()
        assert d <= 1e-12 * ref[s].abs().max().item(), (s, d)
        assert all(np.all(np.isfinite(m.cpu().numpy())) for m in M.values())
