// ps_quickpol.cu -- the QuickPol beam-coupling matrix Xi on the GPU (FP64).
//
// Replaces the loop of quickpolXi! (src/beam.jl:72-109): for l'' = 2..lmax and
// l in the band [l'' - bl, l'' + bu] (l >= 2),
//     Xi[l'', l] = (-1)^(s1+s2+nu1+nu2) sum_l' W[l'] f1(l') f2(l'),
//     f_k(l') = (l' l l''; s_k+nu_k, -s_k, -nu_k) = (l l'' l'; -s_k, -nu_k, s_k+nu_k),
// summed over the common support of the two families (Xisum, src/beam.jl:17-28).
//
// One thread per (l'', l).  Both families follow the general Schulten-Gordon
// recurrence in j = l' (arbitrary m), forward from each family's own jmin and
// backward from the common jmax, and are matched at one common point jm (the
// larger of the two families' midpoints), so the product sum splits into a
// forward part and a backward part with scale lambda1 * lambda2.  Nothing is
// stored; the families stay in registers.
//
// Scaled recurrence.  Divided by j (j + 1), the relation reads
//     a(j+1) f(j+1) + b(j) f(j) + a(j) f(j-1) = 0,   a(j)^2 = P(j) (1 - m3^2 / j^2),
//     b(j) = (2j + 1) ((m2 - m1) - m3 (l - l'') (l + l'' + 1) / (j (j + 1)))
// with the P of the (0 0 0) family.  So with tau the squared (0 0 0) value in the
// factors of ps_plain_fp64.cu and mu(j) = C(j - |m3|) C(j + |m3|) / C(j)^2, for
// which mu(j) mu(j + 1) (1 - m3^2 / (j + 1)^2) = 1, the scaled values
// h = f / sqrt(tau mu) obey
//     h(j + 1) = -((pi / 2) b(j) tau mu h(j) + h(j - 1)):
// no square root and no division.  mu, the two parts of (pi / 2) b and W (times
// sqrt(mu1 mu2)) are tables over j, built per call.  Equal spins (s1 = s2, nu1 = nu2)
// give equal families: one is run.
//
// Bound: the FP64 pipe (see ps_plain_fp64.cu).  FP64 instructions per point: 10 for one
// family (tau 3, mu, b, h, two products, two sums), 8 when m3 = 0, 17 for two; the
// recurrence this replaced took a square root and a division per family and point.
// Measured with it and now, 1000 x 1000 with band (100, 100), as a whole host call:
// 26.9 -> 4.4 ms for nu = 0, s = 2 (one family), 26.7 -> 6.8 ms for nu = -1, 2, s = -2, 2.
#include "ps_internal.cuh"

namespace ps {

namespace {

struct QpParams {
    int lmax, bl, bu;
    int m1[2], m2[2], m3[2];
    HalfTable half;
    // over j = 0 .. 2 lmax + 1
    const double* mu[2];
    const double* e1[2];  // (pi / 2) (2j + 1) (m2 - m1)
    const double* e2[2];  // -(pi / 2) (2j + 1) m3 / (j (j + 1))
    const double* G;      // W sqrt(mu1 mu2), zero beyond W
    double sign;
    double* Xi;
    long long ldx;
};
constexpr int kQpTables = 7;

// The tables over j: mu, e1, e2 of both families, then G.
__global__ void k_quickpol_tables(const QpParams p, double* __restrict__ t, const double* __restrict__ W, int nW, int n)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    double mu[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int m = abs(p.m3[k]);
        const double c = __ldg(p.half.C + j), w = 0.25 * __ldg(p.half.W + j);  // w = (pi / 2) (2j + 1)
        // 0 below the family's support: values there are never used, and j - m is no index
        mu[k] = m == 0 ? 1.0 : (j < m ? 0.0 : __ldg(p.half.C + (j - m)) * __ldg(p.half.C + min(j + m, p.half.top)) / (c * c));
        t[(size_t)(3 * k) * n + j] = mu[k];
        t[(size_t)(3 * k + 1) * n + j] = w * (double)(p.m2[k] - p.m1[k]);
        t[(size_t)(3 * k + 2) * n + j] = j == 0 ? 0.0 : -w * (double)p.m3[k] / ((double)j * (j + 1.0));
    }
    t[(size_t)6 * n + j] = j < nW ? W[j] * (p.m3[0] == p.m3[1] || p.m3[0] == -p.m3[1] ? mu[0] : sqrt(mu[0] * mu[1])) : 0.0;
}

// One family's state in a sweep: the scaled value at the current point and the one before, and
// the normalisation sum over 2 pi (2j + 1) f^2.
struct Sweep {
    double h, hp, N;
};

// SAME: the two families are one.  HASM: some m3 is not 0.
template <bool SAME, bool HASM>
__global__ void __launch_bounds__(128) k_quickpol_fp64(const QpParams p)
{
    // one thread per band element (l'', l), numbered row by row from the top
    // (the longest families first) so that every warp is full
    constexpr int NF = SAME ? 1 : 2;
    const int width = p.bl + p.bu + 1;
    const long long pidx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (pidx >= (long long)(p.lmax - 1) * width) return;
    const int lpp = p.lmax - (int)(pidx / width);  // row l''
    const int l = lpp - p.bl + (int)(pidx % width);
    if (l < 2 || l > p.lmax) return;
    const int lo = min(l, lpp), hi = max(l, lpp), d = hi - lo, jmax = lo + hi;
    const double ds = (double)(l - lpp) * (double)(l + lpp + 1);
    int jmin[NF], jm = 0;
    bool any_zero = false;
#pragma unroll
    for (int k = 0; k < NF; ++k) {
        jmin[k] = max(d, abs(p.m3[k]));
        any_zero |= abs(p.m1[k]) > l || abs(p.m2[k]) > lpp || jmin[k] > jmax;
        jm = max(jm, (jmin[k] + jmax) / 2);
    }
    double xi = 0.0;
    if (!any_zero) {
        if (jm >= jmax) jm = jmax - 1;
        bool fwd[NF];
        int jlo = jm + 1, jstop = jm + 1;
#pragma unroll
        for (int k = 0; k < NF; ++k) {
            fwd[k] = jmin[k] <= jm;
            jlo = min(jlo, fwd[k] ? jmin[k] : jm + 1);
            jstop = min(jstop, fwd[k] ? jm + 1 : jmin[k]);
        }
        const double *Ca = p.half.C - d, *Cb = p.half.C + (2 * lo + d), *Cc = p.half.C + d, *Uc = p.half.U + (2 * hi - d);
        auto tau = [&](int j) {  // t = j - d: C(t) C(2 lo - t) C(t + 2d) / (C(2 hi + t) (2 hi + t + 1))
            return (__ldg(Ca + j) * __ldg(Cb - j)) * (__ldg(Cc + j) * __ldg(Uc + j));
        };
        // one point: the sums over the families' values v (h, or 0 outside the part a sweep sums), then h on
        auto point = [&](int j, Sweep (&s)[NF], const bool (&in)[NF], double& S) {
            const double t = tau(j), w = __ldg(p.half.W + j), g = __ldg(p.G + j);
            double v[NF], tv[NF];
#pragma unroll
            for (int k = 0; k < NF; ++k) {
                const double th = t * s[k].h, q = HASM ? th * __ldg(p.mu[k] + j) : th;
                v[k] = in[k] ? s[k].h : 0.0;
                tv[k] = th;
                s[k].N = fma(w, q * v[k], s[k].N);
                if (SAME) S = fma(g, th * v[0], S);
                const double e1 = __ldg(p.e1[k] + j);
                const double next = -fma(HASM ? fma(__ldg(p.e2[k] + j), ds, e1) : e1, q, s[k].hp);
                s[k].hp = s[k].h;
                s[k].h = next;
            }
            if (!SAME) S = fma(g * tv[0], in[0] ? v[NF - 1] : 0.0, S);
        };
        Sweep F[NF], B[NF];
        double SF = 0.0, SB = 0.0;
        bool on[NF];
#pragma unroll
        for (int k = 0; k < NF; ++k) {
            F[k] = Sweep{0.0, 0.0, 0.0};
            B[k] = Sweep{1.0, 0.0, 0.0};
            on[k] = true;  // a forward family is 0 before its jmin
        }
        for (int j = jlo; j <= jm; ++j) {
#pragma unroll
            for (int k = 0; k < NF; ++k)
                if (j == jmin[k]) {
                    F[k].h = 1.0;
                    F[k].hp = 0.0;
                }
            point(j, F, on, SF);
        }
        // now F.hp = h(jm), F.h = h(jm + 1) of the forward families
        double b0[NF], b1[NF];  // the backward h at jm and jm + 1
        for (int j = jmax; j >= jstop; --j) {
#pragma unroll
            for (int k = 0; k < NF; ++k) on[k] = j >= (fwd[k] ? jm + 1 : jmin[k]);
            point(j, B, on, SB);
            if (j == jm + 1) {
#pragma unroll
                for (int k = 0; k < NF; ++k) {
                    b1[k] = B[k].hp;
                    b0[k] = B[k].h;
                }
            }
        }
        // ---- match, normalise, sign ----
        double lam[NF], N[NF], sg = 1.0;
#pragma unroll
        for (int k = 0; k < NF; ++k) {
            lam[k] = 1.0;
            if (fwd[k]) {
                const double t0 = tau(jm) * (HASM ? __ldg(p.mu[k] + jm) : 1.0);
                const double t1 = tau(jm + 1) * (HASM ? __ldg(p.mu[k] + jm + 1) : 1.0);
                lam[k] = (F[k].hp * b0[k] * t0 + F[k].h * b1[k] * t1) / (b0[k] * b0[k] * t0 + b1[k] * b1[k] * t1);
            }
            N[k] = fma(lam[k] * lam[k], B[k].N, F[k].N);
            // Condon-Shortley: sgn f(jmax) = (-1)^(l - l'' - m3); the matched family has f(jmax) = lambda
            const double cs = ((l - lpp - p.m3[k]) & 1) ? -1.0 : 1.0;
            sg *= lam[k] < 0.0 ? -cs : cs;
        }
        constexpr double kTwoPi = 6.283185307179586477;  // the sums N carry it
        if (SAME) xi = fma(lam[0] * lam[0], SB, SF) * kTwoPi / N[0];
        else xi = fma(lam[0] * lam[NF - 1], SB, SF) * sg * kTwoPi * rsqrt(N[0] * N[NF - 1]);
    }
    p.Xi[(long long)lpp + (long long)l * p.ldx] = p.sign * xi;
}

}  // namespace

size_t quickpol_scratch(int lmax) { return (size_t)kQpTables * (2 * (size_t)lmax + 2); }

cudaError_t launch_quickpol(const double* W, long long nW, int lmax, int bl, int bu, int nu1, int nu2, int s1, int s2,
                            double* Xi, long long ldx, const HalfTable& half, double* scratch, cudaStream_t s)
{
    if (lmax < 2) return cudaSuccess;
    // a band wider than the grid covers the same elements as one of width lmax
    QpParams p;
    p.lmax = lmax;
    p.bl = bl < lmax ? bl : lmax;
    p.bu = bu < lmax ? bu : lmax;
    p.m1[0] = -s1, p.m2[0] = -nu1, p.m3[0] = s1 + nu1;
    p.m1[1] = -s2, p.m2[1] = -nu2, p.m3[1] = s2 + nu2;
    p.half = half;
    const int n = 2 * lmax + 2;
    for (int k = 0; k < 2; ++k) {
        p.mu[k] = scratch + (size_t)(3 * k) * n;
        p.e1[k] = scratch + (size_t)(3 * k + 1) * n;
        p.e2[k] = scratch + (size_t)(3 * k + 2) * n;
    }
    p.G = scratch + (size_t)6 * n;
    p.sign = ((s1 + s2 + nu1 + nu2) & 1) ? -1.0 : 1.0;
    p.Xi = Xi;
    p.ldx = ldx;
    k_quickpol_tables<<<(n + 127) / 128, 128, 0, s>>>(p, scratch, W, (int)nW, n);
    if (cudaError_t e = cudaGetLastError()) return e;
    const int width = p.bl + p.bu + 1;
    const long long total = (long long)(lmax - 1) * width;  // < 2^31 for lmax <= 16383
    const unsigned blocks = (unsigned)((total + 127) / 128);
    const bool same = s1 == s2 && nu1 == nu2, hasm = p.m3[0] != 0 || p.m3[1] != 0;
    // Two blocks, two warps per quarter of an SM, keep its FP64 pipe busy (64 cycles an instruction); the fewer share
    // it, the sooner the longest rows, which come first, are done and the better the rest spread over the SMs.
    // Equal spins, band 201, as many blocks as fit and 2: lmax 300 656 and 515 us, 723 2915 and 2268, 999 4574 and
    // 4368, 1999 17.60 and 17.37 ms (1: 19.2).
    const size_t pad = blocks > 2 * kSMs ? pad_smem(2, 0) : 0;
    auto go = [&](void (*kernel)(QpParams)) -> cudaError_t {
        if (cudaError_t e = allow_smem(kernel, pad)) return e;
        kernel<<<blocks, 128, pad, s>>>(p);
        return cudaGetLastError();
    };
    if (same) return hasm ? go(k_quickpol_fp64<true, true>) : go(k_quickpol_fp64<true, false>);
    return hasm ? go(k_quickpol_fp64<false, true>) : go(k_quickpol_fp64<false, false>);
}

}  // namespace ps
