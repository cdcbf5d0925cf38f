"""Batches whose groups read the table of square-root ratios and slices from tables, and whose groups do not: every
slot of every problem against the allocation-free entry point, which has neither (same arithmetic, so 1e-12 of the
largest entry; differences are those of the last FP64 steps).
"""
import ctypes

import pytest

from test_zz_no_alloc import _noalloc_fn

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _check(ctx, sizes, cases, K, **kw):
    from powerspectra_gpu import synthetic as syn
    fn, L = _noalloc_fn()
    probs, keep = [], []
    for i, lmax in enumerate(sizes):
        n, cs = lmax + 1, cases[i % len(cases)]
        W = [torch.tensor(syn.mask_spectrum(n, 0.5, n / 3.0 + 2.0, seed=7 * i + k), device="cuda") for k in range(K)]
        M = torch.zeros((K, 4, n, n), dtype=torch.float64, device="cuda")
        keep.append((W, M, cs, n))
        probs.append({"lmin": 0, "lmax": lmax, "cases": cs, "nW": n, "ldm": n, "W": [w.data_ptr() for w in W],
                      "M": [M[k, s].data_ptr() for k in range(K) for s in range(4)]})
    torch.cuda.synchronize()
    ctx.batch_prepare(probs, **kw)
    ctx.batch_run()
    torch.cuda.synchronize()
    for W, M, cs, n in keep:
        for k in range(K):
            ref = torch.zeros((4, n, n), dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            assert fn(cs, L.dptr_array([W[k].data_ptr()] * 4), n, 0, n - 1, L.dptr_array([ref[s].data_ptr() for s in range(4)]),
                      n, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
            torch.cuda.synchronize()
            for s in range(4):
                if cs >> s & 1:
                    d = (M[k, s] - ref[s]).abs().max().item()
                    assert d <= 1e-12 * ref[s].abs().max().item(), (n, cs, k, s, d)
                else:
                    assert not bool(M[k, s].any())


MIX = [0xF, 0xC, 0x2, 0x4, 0x8, 0x1]


@pytest.mark.parametrize("gs", [2, 4, 8])
@pytest.mark.parametrize("sizes,K", [(range(299, 347), 1), (range(400, 412), 3)])  # long queues: tables
def test_long_queue(ctx, sizes, K, gs):
    _check(ctx, sizes, MIX, K, group_slots=gs)


@pytest.mark.parametrize("gs", [4, 8])
def test_short_tasks_and_few_problems(ctx, gs):  # no ratios, slices for some
    _check(ctx, [1, 2, 30, 31, 33, 63, 64, 95, 127, 128, 129] * 9, MIX, 1, group_slots=gs)
    _check(ctx, [700, 127, 300], MIX[:3], 2, group_slots=gs)
    for edge, K in ((300, 2), (192, 4), (128, 8)):  # slices of the (0 0 0) family alone
        _check(ctx, [edge - 1, edge], [0x1], K, group_slots=gs)


@pytest.mark.parametrize("sizes", [[40] * 3, list(range(60, 72)), [530, 90, 20]])  # without and with ratios
def test_launch_form(ctx, sizes):
    _check(ctx, sizes, MIX, 2, blocks_per_sm=-1)
