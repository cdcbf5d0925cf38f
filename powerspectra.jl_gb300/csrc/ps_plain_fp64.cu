// ps_plain_fp64.cu -- the plain FP64 coupling kernel.
//
// Replaces the per-pair work of inner_mcm00!/02!/++!/--! (src/modecoupling.jl:78-159)
// and of loop_cov*! (src/covariance.jl:92-446): for every (l1 <= l2) pair the 3j
// families (l1 l2 l3; 0 0 0) and (l1 l2 l3; -2 2 0) are generated in registers
// and contracted with the windows on the fly.  No 3j value is ever stored.
//
// Mapping: one warp owns 32 consecutive l2 of one l1 row (the tiled task list of
// ps_tiles.h: four rows per block).  Every lane's family has the same length
// 2 l1 + 1, so the lanes run in lockstep.
//
// Families.  With t counting the points (l3 = j = d + t from j = d = l2 - l1 to l1 + l2),
// the squared (0 0 0) value is
//     tau(t) = C(t) C(2 l1 - t) C(v - 2 l1) / (C(v) (v + 1)),   v = 2 l2 + t,
//     C(n) = Gamma((n + 1) / 2) / (sqrt(pi) Gamma(n / 2 + 1)),
// the closed form of the (0 0 0) symbol (Edmonds, Angular Momentum in Quantum
// Mechanics, eq. 3.7.17) with the factorial ratios (2m)! / (4^m m!^2) = C(2m)
// continued to odd t.  From C(n) C(n + 1) = 2 / (pi (n + 1)) it follows that
//     tau(t) tau(t + 1) P(j + 1) = (2 / pi)^2,   P(j) = (j^2 - d^2) ((l1 + l2 + 1)^2 - j^2),
// for even and odd t alike.  So the (2 -2 0) family f, which obeys the
// Schulten-Gordon relation a(j+1) f(j+1) + 4 (2j+1) f(j) + a(j) f(j-1) = 0 with
// a^2 = P, is f = sqrt(tau) h with
//     h(t + 1) = -(2 pi (2j + 1) tau(t) h(t) + h(t - 1)):
// no square root, no division, and with q = tau h the three products the
// windows need are at hand, f00^2 = tau, f22^2 = q h, f00 f22 = +-q (f00 changes
// sign from one even point to the next).  At j = d both families have closed
// forms (one term of the Racah sum) of one sign, h(0)^2 = r1 / r2 with
// r = l (l - 1) / ((l + 1)(l + 2)), so there is nothing to match or to
// normalise, and the sweep ends where the windows do (p.nw).
//
// tau factors into A(t) = C(t) C(2 l1 - t), the same for every lane of a row, and
// B(v) = C(v - 2 l1) / (C(v) (v + 1)).  Per 32 points a warp puts A and the B values
// its lanes meet into shared memory (one product per 32 lanes and value); C and
// 1 / (C(v) (v + 1)) come from a table that the context keeps (HalfTable, correctly
// rounded, so no error accumulates in tau).
//
// Bound: GB300's FP64 pipe (2 lanes per cycle and SM, measured 1.06 TFLOP/s),
// which a warp instruction holds for 16 cycles; loads and integer work hide
// behind it.  FP64 instructions per two points with all spin cases: 12 (tau, q,
// h twice, two f22^2, four windows), where the square-root recurrence this
// replaced took about 48 with its 1/sqrt, the normalisation sums and the
// integer-to-double conversions.  Measured with it, with this form in two sweeps
// that meet in the middle, and now: all spin cases at lmax 1999, lmin 2, nW 3999
// 123.7, 34.9 and 32.1 ms; a whole host call (nW = lmax + 1, so that a quarter of the family lies beyond
// the windows), TT at lmax 95 130, 47 and 44 us, EE/BB at lmax 767 8.0, 3.0 and 2.8 ms (1.45
// with its blocks copied whole and fewer blocks per SM, below).  Errors against 128-bit
// arithmetic are smaller than the recurrence's (lmax 2000, all points: 7e-15 at
// most, 1.5e-14 before).
#include "ps_internal.cuh"
#include "ps_epilogue.cuh"

#include <type_traits>

namespace ps {
namespace {

constexpr int kPts = 32;   // points between refills of the shared factors
constexpr int kHalf = 64;  // B ring: entries per parity of v (32 lanes x 32 points meet 47)

struct Factors {
    double A[kPts];
    double B[2][kHalf];  // by parity of v
};

// C(n) and 1 / (C(n) (n + 1)) for any n: indices outside the table belong to lanes that hold no pair
__device__ __forceinline__ double tab_at(const double* __restrict__ t, int n, int top)
{
    return __ldg(t + min(max(n, 0), top));
}
__device__ __forceinline__ void put_b(const CouplingParams& p, Factors& fc, int v, int l1)
{
    fc.B[v & 1][(v >> 1) & (kHalf - 1)] = tab_at(p.half.C, v - 2 * l1, p.half.top) * tab_at(p.half.U, v, p.half.top);
}
__device__ __forceinline__ double flip(double x, int neg)  // -x where neg
{
    return __hiloint2double(__double2hiint(x) ^ (neg << 31), __double2loint(x));
}

// The windows of a launch by what they are contracted with: f00^2, f00 f22, and f22^2 at the even, the
// odd or all points.  A predicated-off FP64 instruction holds the pipe like an executed one (all spin
// cases at lmax 1999 in two sweeps: 66.1 ms with run-time window lists, 34.9 ms with these forms), so the kernels fix
// the number of windows per class at compile time (kForms); a slot without a window repeats another's
// values and its sum is dropped.
enum Class : int { C00, C02, C22E, C22O, C22A, kClasses };
struct PlainParams {
    CouplingParams c;
    const double* w[kClasses][kMaxWin];
    signed char to[kClasses][kMaxWin];  // the window's index in c.win, or -1
};

template <int N00, int N02, int N22E, int N22O, int N22A>
struct Sums {
    double s00[N00 + 1], s02[N02 + 1], se[N22E + 1], so[N22O + 1], sa[N22A + 1];  // + 1: no empty arrays
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int k = 0; k < N00; ++k) s00[k] = 0.0;
#pragma unroll
        for (int k = 0; k < N02; ++k) s02[k] = 0.0;
#pragma unroll
        for (int k = 0; k < N22E; ++k) se[k] = 0.0;
#pragma unroll
        for (int k = 0; k < N22O; ++k) so[k] = 0.0;
#pragma unroll
        for (int k = 0; k < N22A; ++k) sa[k] = 0.0;
    }
    // A point with l1 + l2 + l3 even: tau = f00^2, q = tau h, f22 = sqrt(tau) h; neg: f00 < 0
    __device__ __forceinline__ void even(const PlainParams& p, double tau, double q, double h, int neg, int j)
    {
#pragma unroll
        for (int k = 0; k < N00; ++k) s00[k] = fma(tau, __ldg(p.w[C00][k] + j), s00[k]);
        if (N02 > 0) {
            const double x = flip(q, neg);
#pragma unroll
            for (int k = 0; k < N02; ++k) s02[k] = fma(x, __ldg(p.w[C02][k] + j), s02[k]);
        }
        if (N22E + N22A > 0) {
            const double x = q * h;
#pragma unroll
            for (int k = 0; k < N22E; ++k) se[k] = fma(x, __ldg(p.w[C22E][k] + j), se[k]);
#pragma unroll
            for (int k = 0; k < N22A; ++k) sa[k] = fma(x, __ldg(p.w[C22A][k] + j), sa[k]);
        }
    }
    __device__ __forceinline__ void odd(const PlainParams& p, double q, double h, int j)
    {
        if (N22O + N22A > 0) {
            const double x = q * h;
#pragma unroll
            for (int k = 0; k < N22O; ++k) so[k] = fma(x, __ldg(p.w[C22O][k] + j), so[k]);
#pragma unroll
            for (int k = 0; k < N22A; ++k) sa[k] = fma(x, __ldg(p.w[C22A][k] + j), sa[k]);
        }
    }
    // (this + o) / 4 pi into Xi, each sum to its window; the (2 -2 0) family vanishes for l1 < 2
    __device__ __forceinline__ void give(const PlainParams& p, const Sums& o, int l1, double* Xi) const
    {
        const double u = l1 < 2 ? 0.0 : kInv4Pi;
#pragma unroll
        for (int i = 0; i < kMaxWin; ++i) {
            Xi[i] = 0.0;
#pragma unroll
            for (int k = 0; k < N00; ++k)
                if (p.to[C00][k] == i) Xi[i] = (s00[k] + o.s00[k]) * kInv4Pi;
#pragma unroll
            for (int k = 0; k < N02; ++k)
                if (p.to[C02][k] == i) Xi[i] = l1 < 2 ? 0.0 : (s02[k] + o.s02[k]) * u;
#pragma unroll
            for (int k = 0; k < N22E; ++k)
                if (p.to[C22E][k] == i) Xi[i] = l1 < 2 ? 0.0 : (se[k] + o.se[k]) * u;
#pragma unroll
            for (int k = 0; k < N22O; ++k)
                if (p.to[C22O][k] == i) Xi[i] = l1 < 2 ? 0.0 : (so[k] + o.so[k]) * u;
#pragma unroll
            for (int k = 0; k < N22A; ++k)
                if (p.to[C22A][k] == i) Xi[i] = l1 < 2 ? 0.0 : (sa[k] + o.sa[k]) * u;
        }
    }
};

// The (2 -2 0) family, and the (0 0 0) one with it, over the points t = 0 .. n.  Even and odd points
// alternate between two sets of sums.
template <class S>
__device__ __forceinline__ void sweep22(const PlainParams& P, Factors& fc, int l1, int l2_0, int l2, int n, int lane,
                                        S& S0, S& S1)
{
    const CouplingParams& p = P.c;
    const int d = l2 - l1;
    const double r1 = l1 >= 2 ? (double)l1 * (l1 - 1) / ((double)(l1 + 1) * (l1 + 2)) : 0.0;
    const double r2 = l2 >= 2 ? (double)l2 * (l2 - 1) / ((double)(l2 + 1) * (l2 + 2)) : 1.0;
    double h = sqrt(r1 / r2), hp = 0.0;  // |m| = 2 > l1: h = 0 throughout
    for (int e = lane; e < 96; e += 32) put_b(p, fc, 2 * l2_0 + e, l1);
    auto point = [&](auto even, int t, int neg, S& sum) {
        constexpr bool E = decltype(even)::value;
        const int j = d + t;
        const double tau = fc.A[t & (kPts - 1)] * fc.B[!E][((2 * l2 + t) >> 1) & (kHalf - 1)], q = tau * h;
        if constexpr (E) sum.even(P, tau, q, h, neg, j);
        else sum.odd(P, q, h, j);
        const double next = -fma(__ldg(p.half.W + j), q, hp);
        hp = h;
        h = next;
    };
    const std::true_type even;
    const std::false_type odd;
    for (int t0 = 0; t0 <= n; t0 += kPts) {
        __syncwarp();
        const int ta = t0 + lane;
        fc.A[lane] = tab_at(p.half.C, ta, p.half.top) * tab_at(p.half.C, 2 * l1 - ta, p.half.top);
        if (t0 > 0) put_b(p, fc, 2 * l2_0 + t0 + 62 + lane, l1);  // the other 62 were there before
        __syncwarp();
        const int end = min(t0 + kPts, n + 1);
        int t = t0;
        for (; t + 3 < end; t += 4) {
            point(even, t, 0, S0);
            point(odd, t + 1, 0, S0);
            point(even, t + 2, 1, S1);
            point(odd, t + 3, 0, S1);
        }
        if (t < end) point(even, t, 0, S0);
        if (t + 1 < end) point(odd, t + 1, 0, S0);
        if (t + 2 < end) point(even, t + 2, 1, S1);
    }
}

// The (0 0 0) family alone: tau at every second point t <= n2, no recurrence.  Point n has t = 2n; A
// and B by n = t / 2 and v / 2 = l2 + n.  Two sets of sums keep two chains.
template <class S>
__device__ __forceinline__ void points00(const PlainParams& P, Factors& fc, int l1, int l2_0, int l2, int n2, int lane,
                                         S& S0, S& S1)
{
    const CouplingParams& p = P.c;
    const int d = l2 - l1;
    put_b(p, fc, 2 * (l2_0 + lane), l1);
    for (int n0 = 0; 2 * n0 <= n2; n0 += kPts) {
        __syncwarp();
        const int ta = 2 * (n0 + lane);
        fc.A[lane] = tab_at(p.half.C, ta, p.half.top) * tab_at(p.half.C, 2 * l1 - ta, p.half.top);
        put_b(p, fc, 2 * (l2_0 + n0 + 32 + lane), l1);
        __syncwarp();
        const int end = min(n0 + kPts, n2 / 2 + 1);
        int n = n0;
#pragma unroll 2
        for (; n + 1 < end; n += 2) {
            S0.even(P, fc.A[n - n0] * fc.B[0][(l2 + n) & (kHalf - 1)], 0.0, 0.0, 0, d + 2 * n);
            S1.even(P, fc.A[n + 1 - n0] * fc.B[0][(l2 + n + 1) & (kHalf - 1)], 0.0, 0.0, 0, d + 2 * n + 2);
        }
        if (n < end) S0.even(P, fc.A[n - n0] * fc.B[0][(l2 + n) & (kHalf - 1)], 0.0, 0.0, 0, d + 2 * n);
    }
}

struct __align__(16) PlainSmem {
    Factors f[kWarpsPerBlock];
    double stage[kWarpsPerBlock][kMaxWin * 32];
    TileRows rows;
};
template <int N00, int N02, int N22E, int N22O, int N22A>
__global__ void __launch_bounds__(kWarpsPerBlock * 32) k_coupling_fp64(const PlainParams P)
{
    __shared__ PlainSmem sm;
    const CouplingParams& p = P.c;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the task list is tiled: kTileRows tasks per block, rows outside [lmin, lmax] as l1 = -1
    const int gw = (int)(blockIdx.x * (unsigned)kWarpsPerBlock) + warp;
    int2 task = gw < p.ntasks ? p.tasks[gw] : make_int2(-1, 0);
    wait_for_previous(task.x);  // the padded windows
    const int l1 = task.x, l2raw = task.y + lane;
    const bool active = l1 >= 0 && l2raw >= l1 && l2raw <= p.lmax;
    double Xi[kMaxWin];
    if (l1 >= 0) {  // warp-uniform
        const int l2 = min(max(l2raw, l1), p.lmax);  // lanes outside compute values nobody writes
        using S = Sums<N00, N02, N22E, N22O, N22A>;
        S a, b;
        a.zero();
        b.zero();
        // the points whose j a window reaches, for the warp's smallest d (the others' windows end in zeros)
        const int n = min(p.nw - 1 - (max(task.y, l1) - l1), 2 * l1);
        if constexpr (N02 + N22E + N22O + N22A > 0) sweep22(P, sm.f[warp], l1, task.y, l2, n, lane, a, b);
        else points00(P, sm.f[warp], l1, task.y, l2, n, lane, a, b);
        a.give(P, b, l1, Xi);
    }
    write_tile<kMaxWin, true>(p, l1, task.y, active, Xi, &sm.stage[0][0], kMaxWin * 32, sm.rows, warp, lane);
}

struct Form {
    int n[kClasses];
    void (*kernel)(PlainParams);
};
#define PS_FORM(a, b, c, d, e) Form{{a, b, c, d, e}, k_coupling_fp64<a, b, c, d, e>}
// Cheapest first.  They cover the mode-coupling cases of one call (up to one window per class), the
// covariance kinds (8, 4 or 2 windows of one class, TETE's 4 and 1), ps_xi (one class), and the groups
// that ps_mcm_set makes: whole windows (at most 4 of a class when it mixes classes), or ++ and --.
const Form kForms[] = {
    PS_FORM(1, 0, 0, 0, 0), PS_FORM(2, 0, 0, 0, 0), PS_FORM(4, 0, 0, 0, 0), PS_FORM(8, 0, 0, 0, 0),
    PS_FORM(0, 1, 0, 0, 0), PS_FORM(0, 0, 1, 0, 0), PS_FORM(0, 0, 0, 1, 0), PS_FORM(1, 1, 0, 0, 0),
    PS_FORM(0, 0, 1, 1, 0), PS_FORM(0, 0, 0, 0, 1), PS_FORM(0, 4, 0, 0, 0), PS_FORM(1, 0, 1, 1, 0),
    PS_FORM(0, 0, 4, 0, 0), PS_FORM(1, 4, 0, 0, 0), PS_FORM(1, 1, 1, 1, 0), PS_FORM(0, 8, 0, 0, 0),
    PS_FORM(0, 0, 8, 0, 0), PS_FORM(0, 0, 0, 8, 0), PS_FORM(2, 2, 2, 2, 0), PS_FORM(0, 0, 4, 4, 0),
    PS_FORM(0, 0, 8, 8, 0), PS_FORM(0, 0, 0, 0, 8), PS_FORM(4, 4, 4, 4, 0),
};
#undef PS_FORM

}  // namespace

cudaError_t launch_plain_fp64(const CouplingParams& p, cudaStream_t s)
{
    const int threads = kWarpsPerBlock * 32;
    const unsigned blocks = (unsigned)((p.ntasks + kWarpsPerBlock - 1) / kWarpsPerBlock);
    if (blocks == 0) return cudaSuccess;
    PlainParams P;
    P.c = p;
    int n[kClasses] = {0, 0, 0, 0, 0};
    for (int c = 0; c < kClasses; ++c)
        for (int k = 0; k < kMaxWin; ++k) {
            P.w[c][k] = p.win[0].wW;
            P.to[c][k] = -1;
        }
    for (int k = 0; k < p.nwin; ++k) {
        const int pr = p.win[k].product, par = p.win[k].parity;
        if (pr != PROD_22_22 && par == PAR_ODD) continue;  // f00 vanishes at odd points: Xi = 0
        const int c = pr == PROD_00_00 ? C00 : (pr == PROD_00_22 ? C02 : (par == PAR_EVEN ? C22E : (par == PAR_ODD ? C22O : C22A)));
        P.w[c][n[c]] = p.win[k].wW;
        P.to[c][n[c]++] = (signed char)k;
    }
    for (const Form& f : kForms) {
        bool fits = true;
        for (int c = 0; c < kClasses; ++c) fits = fits && n[c] <= f.n[c];
        if (!fits) continue;
        // Blocks that share an SM: one warp per quarter of an SM keeps its FP64 pipe busy for all but the refills
        // (64 cycles an instruction), and the fewer share it, the sooner the longest rows, which come first,
        // are done and the better the rest spread over the SMs.  ++/-- at nW = lmax + 1, with as many as fit (8), 1, 2
        // and 3: lmax 255 (288 blocks) 109, 94, 110, 110 us; 383 (624) 271, 231, 206, 225; 511 (1088) 534, 483, 429,
        // 426; 767 (2400) 1366, 1481, 1301, 1302; 1001 (4224) 2797, 3166, 2772, 2777.  The other forms agree: with TT, 8 TT, TE,
        // 8 TE, all spins of one and two windows and TT and TE of four, at lmax 255 to 1400, the rule is within 3 % of the best
        // of 1, 2, 3, 4 and as many as fit (TT at 383 41.6 us, 51.9 with as many as fit; all spins 220 and 296).
        const int share = blocks <= 2 * kSMs ? 1 : (blocks <= 8 * kSMs ? 2 : 3);
        const size_t pad = blocks > kSMs ? pad_smem(share, sizeof(PlainSmem)) : 0;
        return launch_after(f.kernel, dim3(blocks), dim3(threads), pad, s, P);
    }
    return cudaErrorInvalidValue;
}

// ---------------------------------------------------------------------------
// FMA-pipe probe: 8 independent FMA chains per thread, FMA counted as 2 flops.
template <typename T>
__global__ void __launch_bounds__(256) k_fma_probe(T* sink, int iters)
{
    T a0 = (T)threadIdx.x * (T)1e-3, a1 = a0 + (T)1, a2 = a0 + (T)2, a3 = a0 + (T)3;
    T a4 = a0 + (T)4, a5 = a0 + (T)5, a6 = a0 + (T)6, a7 = a0 + (T)7;
    const T b = (T)0.999999, c = (T)1e-6;
    for (int i = 0; i < iters; ++i) {
        a0 = fma(a0, b, c); a1 = fma(a1, b, c); a2 = fma(a2, b, c); a3 = fma(a3, b, c);
        a4 = fma(a4, b, c); a5 = fma(a5, b, c); a6 = fma(a6, b, c); a7 = fma(a7, b, c);
    }
    T r = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (r == (T)-12345.0) sink[blockIdx.x] = r;  // keeps the chains alive; never true
}

cudaError_t launch_fma_probe(int fp64, double* sink, int blocks, int iters, cudaStream_t s)
{
    if (fp64)
        k_fma_probe<double><<<blocks, 256, 0, s>>>(sink, iters);
    else
        k_fma_probe<float><<<blocks, 256, 0, s>>>((float*)sink, iters);
    return cudaGetLastError();
}

}  // namespace ps
