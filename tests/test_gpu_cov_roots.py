"""The roots in the covariance formulas.

One root per product in FP64: spectra of 1 and 2 only, so that S1(a) S1(b) S2(a) S2(b) is 1, 4 or 16 and its root exact where
the roots of the two pairs are not, and windows of zeros but for one.  An element is then that window's Xi times 1, 2
or 4, to the last bit.

Signs: an element is NaN where a pair of unequal signs enters a root, as in the reference's formulas, and for nothing
else.
"""
import numpy as np
import pytest

from oracle import oracle as o

pytestmark = pytest.mark.gpu

# kind: family product and parity of the windows, (window, the two spectra whose four values share one root)
ROOTS = {"TTTT": ((0, 0), ((0, 0, 1), (1, 2, 3))), "EEEE": ((1, 1), ((0, 0, 1), (1, 2, 3))),
         "TETE": ((2, 1), ((0, 0, 1),))}


@pytest.mark.parametrize("kind", list(ROOTS))
def test_one_root_of_a_product(ctx, kind):
    from powerspectra_gpu import synthetic as syn
    L = 70
    (product, parity), pairs = ROOTS[kind]
    W = syn.mask_spectrum(2 * L + 1, 0.6, 30.0, seed=11)
    zero = np.zeros(2 * L + 1)
    s = np.where(np.arange(L + 1) % 3 == 1, 2.0, 1.0)
    R = [np.ones(L + 1)] * o.COV_NRATIOS[kind]
    nw = o.COV_NWINDOWS[kind]
    for k, i, j in pairs:
        Ws = [W if q == k else zero for q in range(nw)]
        S = [s if q in (i, j) else np.zeros(L + 1) for q in range(4)]
        C = ctx.coupledcov(kind, S, R, Ws, 0, L)
        X = ctx.xi(product, parity, Ws[k:] + Ws[:k], 0, L)[0] if kind != "TETE" else None
        if X is None:  # TETE mixes families: its own element for spectra of ones
            X = ctx.coupledcov(kind, [np.ones(L + 1) if q in (i, j) else S[q] for q in range(4)], R, Ws, 0, L)
        assert np.array_equal(C, np.outer(s, s) * X)


@pytest.mark.parametrize("kind", list(o.COV_KINDS))
@pytest.mark.parametrize("route", ["plain", "chosen", "set"])
def test_signs_zeros_and_infinities(ctx, kind, route):
    torch = pytest.importorskip("torch")
    from powerspectra_gpu import synthetic as syn
    L = 40
    n, nW = L + 1, 2 * L + 1
    rng = np.random.default_rng(5)
    S = [rng.uniform(0.5, 2.0, n) for _ in range(4)]
    for q in range(4):
        S[q][3 + q] *= -1.0
        S[q][10 + q] = 0.0
        S[q][20 + 2 * q:22 + 2 * q] *= -1.0  # equal signs: a positive product
        S[q][30 + q] = np.inf
    R = [rng.uniform(0.5, 2.0, n) for _ in range(o.COV_NRATIOS[kind])]
    Ws = [syn.mask_spectrum(nW, 0.5 + 0.03 * k, 20.0, seed=k) for k in range(o.COV_NWINDOWS[kind])]
    with np.errstate(invalid="ignore", over="ignore"):
        ref = o.loop_cov(kind, S, R, Ws, 0, L)
    if route == "set":  # Xi by the tensor-core kernels or the others, then the blocks from them
        d = lambda xs: [torch.tensor(x, device="cuda") for x in xs]
        dS, dR, dW = d(S), d(R), d(Ws)
        C = torch.zeros((3, n, n), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        p = lambda xs: [x.data_ptr() for x in xs]
        ctx.coupledcov_set_device([(kind, p(dS), p(dR), p(dW), C[b].data_ptr()) for b in range(3)], nW, 0, L, n,
                                  mode="chosen")
        ctx.synchronize()
        got = C[1].cpu().numpy()
    else:
        got = ctx.coupledcov(kind, S, R, Ws, 0, L, mode=route)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    assert np.array_equal(np.isinf(got), np.isinf(ref))
    fin = np.isfinite(ref)
    assert np.array_equal(np.signbit(got[np.isinf(ref)]), np.signbit(ref[np.isinf(ref)]))
    tol = 1e-12 if route == "plain" else 2e-6
    A = o.loop_cov(kind, [np.where(np.isfinite(x), np.abs(x), 0.0) for x in S], R, Ws, 0, L)
    assert np.all(np.abs(got[fin] - ref[fin]) <= tol * np.maximum(np.abs(A[fin]), np.abs(ref[fin])) + 1e-300)
