// ps_cov_epilogue.cuh -- per-pair combination of the Xi_k into a covariance
// element, one formula per loop_cov*! kernel of the reference.
#pragma once

#include "ps_internal.cuh"

namespace ps {

// The FP64 kernels' root.  One function for the six of an element: a kernel of some 100 us runs its epilogue a few times,
// and the code of six inlined roots took longer to arrive than to run (EE x EE at lmax 230 211 us, 187 with the function;
// TT x EE at lmax 700 364 and 355; TE x TE at 230 154 and 155).
static __device__ __noinline__ double root(double x) { return sqrt(x); }

// X[k] are the Xi of windows W1..Wk (already divided by 4pi), Sa, Sb, Ra, Rb the spectra and noise
// ratios at l1 = a and l2 = b, g[i] = sqrt(Sa[i] Sb[i]) for the spectra that need it (cov_roots).
// ONE_ROOT: the root of a product of two such pairs as one root, as the reference takes it, for the FP64 kernels; the
// product of the two roots has two roundings of 1e-16 more, which Xi with the fast arithmetic's 1e-7 do not show (the
// further roots would cost TTTT and EEEE at lmax 700 3 %).  They are taken inside their case: ahead of the
// switch, as predicated instructions or a loop, they cost every kind (TTEE at lmax 700 in FP64 364 -> 377 us).
template <bool ONE_ROOT>
__device__ __forceinline__ double cov_form(int kind, const double* Sa, const double* Sb, const double* g,
                                           const double* Ra, const double* Rb, const double* X)
{
    auto product = [&](int i) {  // of the pairs i and i + 1
        return ONE_ROOT ? root(Sa[i] * Sb[i] * Sa[i + 1] * Sb[i + 1]) : g[i] * g[i + 1];
    };
    switch (kind) {
    case PS_COV_TTTT:
    case PS_COV_EEEE: {  // src/covariance.jl:110-118 (TTTT), :171-179 (EEEE); ip, jq, iq, jp
        const double ip = Ra[0] * Rb[0], jq = Ra[1] * Rb[1], iq = Ra[2] * Rb[2], jp = Ra[3] * Rb[3];
        return product(0) * X[0] + product(2) * X[1] + g[0] * X[2] * jq + g[1] * X[3] * ip + g[2] * X[4] * jp +
               g[3] * X[5] * iq + X[6] * (ip * jq) + X[7] * (iq * jp);
    }
    case PS_COV_TTTE:  // src/covariance.jl:225-230; TTip, TTjp, TEiq, TEjq; r_ip, r_jp
        return (g[0] * (Sa[3] + Sb[3]) * X[0] + g[1] * (Sa[2] + Sb[2]) * X[1] + (Sa[3] + Sb[3]) * X[2] * Ra[0] * Rb[0] +
                (Sa[2] + Sb[2]) * X[3] * Ra[1] * Rb[1]) / 2;
    case PS_COV_TETE: {  // src/covariance.jl:292-297; TTip, EEjq, TEiq, TEjp; r_TT, r_PP
        const double rT = Ra[0] * Rb[0], rP = Ra[1] * Rb[1];
        return product(0) * X[0] + 0.5 * (Sa[2] * Sb[3] + Sa[3] * Sb[2]) * X[1] + g[0] * X[2] * rP + g[1] * X[3] * rT +
               X[4] * (rT * rP);
    }
    case PS_COV_TEEE:
    case PS_COV_TEEE_PLANCK:  // src/covariance.jl:362-367 and :392-397; EEjq, EEjp, TEip, TEiq; r_jq, r_jp
        return (g[0] * (Sa[2] + Sb[2]) * X[0] + g[1] * (Sa[3] + Sb[3]) * X[1] + (Sa[2] + Sb[2]) * X[2] * Ra[0] * Rb[0] +
                (Sa[3] + Sb[3]) * X[3] * Ra[1] * Rb[1]) / 2;
    default:  // PS_COV_TTEE, src/covariance.jl:438-441; TEip, TEiq, TEjq, TEjp
        return ((Sa[0] * Sb[2] + Sa[2] * Sb[0]) * X[0] + (Sa[1] * Sb[3] + Sa[3] * Sb[1]) * X[1]) / 2;
    }
}

// How many spectra of a kind enter through sqrt(Sa Sb): the first ones.
__host__ __device__ constexpr int cov_roots(int kind)
{
    return kind == PS_COV_TTTT || kind == PS_COV_EEEE ? 4 : (kind == PS_COV_TTEE ? 0 : 2);
}
// ... and how many noise ratios it has.
__host__ __device__ constexpr int cov_ratios(int kind)
{
    return kind == PS_COV_TTTT || kind == PS_COV_EEEE ? 4 : (kind == PS_COV_TTEE ? 0 : 2);
}

// The element of one pair (l1 = a, l2 = b), a <= b.
template <bool ONE_ROOT>
__device__ __forceinline__ double cov_combine(int kind, const double* const* S, const double* const* R,
                                              const double* X, int a, int b)
{
    double Sa[4], Sb[4], g[4], Ra[4], Rb[4];
    const int ng = cov_roots(kind), nr = cov_ratios(kind);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        Sa[i] = S[i][a];
        Sb[i] = S[i][b];
        const double p = Sa[i] * Sb[i];
        g[i] = i < ng ? (ONE_ROOT ? root(p) : sqrt(p)) : 0.0;
        Ra[i] = i < nr ? R[i][a] : 0.0;
        Rb[i] = i < nr ? R[i][b] : 0.0;
    }
    return cov_form<ONE_ROOT>(kind, Sa, Sb, g, Ra, Rb, X);
}

}  // namespace ps
