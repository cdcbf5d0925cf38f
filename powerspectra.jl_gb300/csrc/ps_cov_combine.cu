// ps_cov_combine.cu -- a covariance block from Xi matrices computed beforehand.
//
// ps_coupledcov_set_device computes the Xi of every window of the blocks whose
// windows all use the squared (0 0 0) family (TTTT, TTTE, TTEE) in shared
// tensor-core launches, then forms each block here with the same per-element
// formula the fused epilogue of the coupling kernel uses (ps_cov_epilogue.cuh,
// after src/covariance.jl:110-118, :225-230, :438-441).
//
// Xi and C are symmetric, so a block of threads forms one 32 x 32 tile on or above
// the diagonal and writes it and its mirror image: each Xi is read half, and half
// the elements are formed.  The geometric means sqrt(S[l1] S[l2]) are products of
// roots taken once per l and tile, 64 per 1024 elements and spectrum instead of
// 1024 (the kernel was bound by FP64 square roots: six of them per element of
// TTTT and EEEE).  Measured, six blocks at lmax 2508: 3.12 -> 0.78 ms; what bounds it
// now is the FP64 pipe and the one read of the Xi together.
#include "ps_internal.cuh"
#include "ps_cov_epilogue.cuh"

namespace ps {
namespace {

constexpr int kTile = 32, kRows = 8;

// sqrt(|s|) with the sign of s: the product of two is sqrt(s t) for equal signs and negative otherwise
__device__ __forceinline__ double signed_root(double s) { return copysign(sqrt(fabs(s)), s); }
// sqrt(s t) from the signed roots: NaN for unequal signs (as sqrt of a negative number), 0 where one is 0
__device__ __forceinline__ double mean_of(double s, double t)
{
    const double g = s * t;
    return g < 0.0 ? __longlong_as_double(0x7ff8000000000000LL) : g;
}

template <int KIND>
__global__ void __launch_bounds__(kTile * kRows) k_cov_combine(const CovCombineParams p)
{
    const int bi = blockIdx.x, bj = blockIdx.y;  // tile of rows, tile of columns
    if (bi > bj) return;
    constexpr int NG = cov_roots(KIND), NR = cov_ratios(KIND);
    constexpr int NX = KIND == PS_COV_TTTT || KIND == PS_COV_EEEE ? 8 : (KIND == PS_COV_TETE ? 5 : (KIND == PS_COV_TTEE ? 2 : 4));
    __shared__ double sS[2][4][kTile], sG[2][4][kTile], sR[2][4][kTile];  // [rows, columns]
    __shared__ double sC[kTile][kTile + 1];
    const int tx = threadIdx.x, ty = threadIdx.y;
    {
        // thread (tx, ty): l = lane of the row tile (ty < 4) or the column tile, spectrum ty % 4
        const int side = ty >> 2, k = ty & 3, q = (side ? bj : bi) * kTile + tx;
        const bool in = q < p.n;
        const double s = in ? p.S[k][p.lmin + q] : 0.0;
        sS[side][k][tx] = s;
        sG[side][k][tx] = k < NG ? signed_root(s) : 0.0;
        sR[side][k][tx] = in && k < NR ? p.R[k][p.lmin + q] : 0.0;
    }
    __syncthreads();
    const int i = bi * kTile + tx;
    for (int c = ty; c < kTile; c += kRows) {
        const int j = bj * kTile + c;
        double e = 0.0;
        if (i < p.n && j < p.n && i <= j) {
            double x[NX], Sa[4], Sb[4], g[4], Ra[4], Rb[4];
#pragma unroll
            for (int k = 0; k < NX; ++k) x[k] = __ldg(p.X[k] + i + (long long)j * p.ldx);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                Sa[k] = sS[0][k][tx];
                Sb[k] = sS[1][k][c];
                g[k] = k < NG ? mean_of(sG[0][k][tx], sG[1][k][c]) : 0.0;
                Ra[k] = sR[0][k][tx];
                Rb[k] = sR[1][k][c];
            }
            e = cov_form<false>(KIND, Sa, Sb, g, Ra, Rb, x);
            p.C[i + (long long)j * p.ldc] = e;
        }
        sC[c][tx] = e;
    }
    __syncthreads();
    // the mirror image: element (j, i), j along the warp
    const int j = bj * kTile + tx;
    for (int c = ty; c < kTile; c += kRows) {
        const int ir = bi * kTile + c;
        if (ir < p.n && j < p.n && ir < j) p.C[j + (long long)ir * p.ldc] = sC[tx][c];
    }
}

}  // namespace

cudaError_t launch_cov_combine(const CovCombineParams& p, cudaStream_t s)
{
    if (p.n <= 0) return cudaSuccess;
    const unsigned nt = (unsigned)((p.n + kTile - 1) / kTile);
    const dim3 grid(nt, nt), block(kTile, kRows);
    switch (p.kind) {
    case PS_COV_TTTT:
    case PS_COV_EEEE: k_cov_combine<PS_COV_TTTT><<<grid, block, 0, s>>>(p); break;
    case PS_COV_TTTE: k_cov_combine<PS_COV_TTTE><<<grid, block, 0, s>>>(p); break;
    case PS_COV_TETE: k_cov_combine<PS_COV_TETE><<<grid, block, 0, s>>>(p); break;
    case PS_COV_TEEE:
    case PS_COV_TEEE_PLANCK: k_cov_combine<PS_COV_TEEE><<<grid, block, 0, s>>>(p); break;
    default: k_cov_combine<PS_COV_TTEE><<<grid, block, 0, s>>>(p); break;
    }
    return cudaGetLastError();
}

}  // namespace ps
