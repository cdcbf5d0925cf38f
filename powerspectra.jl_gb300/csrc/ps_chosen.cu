// ps_chosen.cu -- launches of the chosen coupling kernel (ps_chosen_task.cuh)
// for window groups of up to 5 slots, and the window preparation kernels.
// Groups of 6-8 slots are instantiated in ps_chosen8.cu, the batched kernel in
// ps_batch_chosen.cu, so the three compile in parallel.
#include "ps_chosen_task.cuh"

namespace ps {

cudaError_t launch_chosen8(const CouplingParams& p, uint32_t spec, bool n00, bool n22, cudaStream_t s);

cudaError_t launch_chosen(const CouplingParams& p, cudaStream_t s)
{
    bool n00 = false, n22 = false;
    for (int k = 0; k < p.nwin; ++k) {
        if (p.win[k].product != PROD_22_22) n00 = true;
        if (p.win[k].product != PROD_00_00) n22 = true;
    }
    const uint32_t spec = spec_of(p);
    const int nw = p.nwin;
    if (p.ntasks <= 0) return cudaSuccess;
    // the smallest instantiation whose slot list starts with this configuration
    if (spec_fits(spec, nw, W00, 1)) return launch_cfg<1, W00>(p, n00, n22, s);
    if (spec_fits(spec, nw, W02, 1)) return launch_cfg<1, W02>(p, n00, n22, s);
    if (spec_fits(spec, nw, WPP, 1)) return launch_cfg<1, WPP>(p, n00, n22, s);
    if (spec_fits(spec, nw, WMM, 1)) return launch_cfg<1, WMM>(p, n00, n22, s);
    if (spec_fits(spec, nw, S_PPMM, 2)) return launch_cfg<2, S_PPMM>(p, n00, n22, s);
    if (spec_fits(spec, nw, rep(W00, 4), 4)) return launch_cfg<4, rep(W00, 4)>(p, n00, n22, s);
    if (spec_fits(spec, nw, S_PPMM2, 4)) return launch_cfg<4, S_PPMM2>(p, n00, n22, s);
    if (spec_fits(spec, nw, S_MCM4, 4)) return launch_cfg<4, S_MCM4>(p, n00, n22, s);
    if (spec_fits(spec, nw, rep(W02, 4), 4)) return launch_cfg<4, rep(W02, 4)>(p, n00, n22, s);
    if (spec_fits(spec, nw, rep(WPP, 4), 4)) return launch_cfg<4, rep(WPP, 4)>(p, n00, n22, s);
    if (spec_fits(spec, nw, rep(WMM, 4), 4)) return launch_cfg<4, rep(WMM, 4)>(p, n00, n22, s);
    if (spec_fits(spec, nw, S_TETE, 5)) return launch_cfg<5, S_TETE>(p, n00, n22, s);
    if (nw <= 1) return launch_cfg<1, 0>(p, n00, n22, s);
    if (nw <= 2) return launch_cfg<2, 0>(p, n00, n22, s);
    if (nw <= 4) return launch_cfg<4, 0>(p, n00, n22, s);
    return launch_chosen8(p, spec, n00, n22, s);
}

// Entry j of a window: (2 l3 + 1) W[l3] in FP64, zero for j >= nW, and split into (float mantissa in
// [0.5, 1), exponent), zeros as (0, kZeroExp).
__device__ __forceinline__ void prep_entry(const double* __restrict__ src, long long nW, int j, double* wW, int2* bf)
{
    const double v = j < nW ? (2.0 * j + 1.0) * src[j] : 0.0;
    wW[j] = v;
    if (!bf) return;
    int e = 0;
    const double m = v == 0.0 ? 0.0 : frexp(v, &e);
    bf[j] = v == 0.0 ? make_int2(0, kZeroExp) : make_int2(__float_as_int((float)m), e);
}

// All windows of a batch in one launch: pad + premultiply + split.
__global__ void k_prep_windows(const WinPrep* __restrict__ list, int n)
{
    const WinPrep w = list[blockIdx.y];
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < w.wlen; j += gridDim.x * blockDim.x)
        prep_entry(w.src, w.nW, j, w.wW, w.bf);
}

// The windows of one call: window blockIdx.y.  One launch instead of one or two per window, which cost
// about 2.5 us each (31 windows of a covariance set: 62 launches).
struct SetPrep {
    const double* src[kSetWindows];
    long long nW;
    double* wW;
    int2* bf;
    int wlen;
};
__global__ void k_prep_set(const SetPrep p)
{
    const int k = blockIdx.y;
    int2* bf = p.bf ? p.bf + (size_t)k * p.wlen : nullptr;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < p.wlen; j += gridDim.x * blockDim.x)
        prep_entry(p.src[k], p.nW, j, p.wW + (size_t)k * p.wlen, bf);
}

cudaError_t launch_prep_set(const double* const* src, int K, long long nW, int wlen, double* wW, int2* bf,
                            cudaStream_t s)
{
    for (int k0 = 0; k0 < K; k0 += kSetWindows) {
        const int n = K - k0 < kSetWindows ? K - k0 : kSetWindows;
        SetPrep p;
        for (int k = 0; k < n; ++k) p.src[k] = src[k0 + k];
        p.nW = nW;
        p.wW = wW + (size_t)k0 * wlen;
        p.bf = bf ? bf + (size_t)k0 * wlen : nullptr;
        p.wlen = wlen;
        int bx = (wlen + 255) / 256;
        if (bx > 64) bx = 64;
        k_prep_set<<<dim3(bx, n), 256, 0, s>>>(p);
        if (cudaError_t e = cudaGetLastError()) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_prep_windows(const WinPrep* list, int n, int max_wlen, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    int threads = 256;
    int bx = (max_wlen + threads - 1) / threads;
    if (bx > 64) bx = 64;
    k_prep_windows<<<dim3(bx, n), threads, 0, s>>>(list, n);
    return cudaGetLastError();
}

}  // namespace ps
