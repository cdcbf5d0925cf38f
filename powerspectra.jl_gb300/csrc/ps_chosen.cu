// ps_chosen.cu -- launches of the chosen coupling kernel (ps_chosen_task.cuh)
// for window groups of up to 5 slots, and the window preparation kernels.
// Groups of 6-8 slots are instantiated in ps_chosen8.cu, the batched kernel in
// ps_batch_chosen.cu, so the three compile in parallel.
#include "ps_chosen_task.cuh"

namespace ps {

cudaError_t launch_chosen8(const CouplingParams& p, uint32_t spec, bool n00, bool n22, cudaStream_t s);

namespace {

// The instantiations: a launch takes the first whose slot list starts with its configuration, or the one
// of its number of slots that reads the configuration from the parameters.
struct Inst {
    uint32_t spec;
    int n;  // slots
    bool coef;  // reads the table of square-root ratios
    cudaError_t (*launch)(const CouplingParams&, bool, bool, cudaStream_t);
};
#define PS_INST(n, spec) Inst{spec, n, kHasCoef<n, spec>, launch_cfg<n, spec>}
const Inst kInst[] = {
    PS_INST(1, W00),          PS_INST(1, W02),          PS_INST(1, WPP),          PS_INST(1, WMM),
    PS_INST(2, S_PPMM),       PS_INST(4, rep(W00, 4)),  PS_INST(4, S_PPMM2),      PS_INST(4, S_MCM4),
    PS_INST(4, rep(W02, 4)),  PS_INST(4, rep(WPP, 4)),  PS_INST(4, rep(WMM, 4)),  PS_INST(5, S_TETE),
};
const Inst kAny[] = {PS_INST(1, 0), PS_INST(2, 0), PS_INST(4, 0)};
#undef PS_INST

const Inst* find_inst(const CouplingParams& p, uint32_t spec)  // null: launch_chosen8
{
    for (const Inst& i : kInst)
        if (spec_fits(spec, p.nwin, i.spec, i.n)) return &i;
    for (const Inst& i : kAny)
        if (p.nwin <= i.n) return &i;
    return nullptr;
}

}  // namespace

bool has_coef(const CouplingParams& p)
{
    const Inst* i = find_inst(p, spec_of(p));
    return i && i->coef;
}
// In a call by itself: below lmax 512 the copies of a warp's first chunk wait longer than its square roots take (TT, TE
// and ++/-- together, without and with the table: lmax 95 55.8 and 55.6 us, ++ alone 38.0 and 43.3; 383 83.7 and 84.8;
// 767 268.0 and 258.5).  In a row of launches it gains at any lmax (200 of 20-200: 3432 and 3214 us).
bool reads_coef(const CouplingParams& p) { return p.lmax >= 512 && has_coef(p); }

size_t slice_table_bytes(const CouplingParams& p)
{
    const Inst* i = find_inst(p, spec_of(p));
    return slice_bytes(i ? i->n : 8) * (size_t)slice_count(p.lmax);
}
size_t slice_table_most(int lmax) { return slice_bytes(8) * (size_t)slice_count(lmax); }

namespace {

// One row of the table per blockIdx.y.
__global__ void __launch_bounds__(256) k_coef(float4* __restrict__ t, int lmax)
{
    const int l1 = blockIdx.y, i = blockIdx.x * 256 + threadIdx.x;
    const long long n = coef_row(lmax, lmax + 1), row = coef_row(lmax, l1);
    const float h = (float)(2 * l1 + 1);
    auto put = [](float4* at, ff rho, ff r) { *at = make_float4(rho.h, rho.l, r.h, r.l); };
    if (i < 2 * lmax + 160 - l1) {
        ff rho = ff_make(0.0f), r = rho;
        const float a = (float)(i - 62);
        if (a >= 0.0f) sqrt_ratio(two_prod(a, a + h), two_prod(a + 1.0f, a + h + 1.0f), rho, r);
        put(t + row + i, ff_neg(rho), r);
        const float b = (float)(i + l1 - 92);
        rho = r = ff_make(0.0f);
        if (b > 0.0f) sqrt_ratio(two_prod(b + 1.0f, b + h + 1.0f), two_prod(b, b + h), rho, r);
        put(t + n + row + i, ff_neg(rho), r);
    }
    if (i < l1 || (l1 == lmax && i < l1 + 32)) {
        ff rho = ff_make(0.0f), r = rho;
        const float x = (float)i;
        if (i < l1) sqrt_ratio(two_prod(x, h - x), two_prod(x + 1.0f, h - 1.0f - x), rho, r);
        put(t + 2 * n + coef_row_g(l1) + i, rho, r);
    }
}

}  // namespace

cudaError_t launch_coef(float4* t, int lmax, cudaStream_t s)
{
    k_coef<<<dim3((unsigned)((2 * lmax + 160 + 255) / 256), (unsigned)(lmax + 1)), 256, 0, s>>>(t, lmax);
    return cudaGetLastError();
}

cudaError_t launch_chosen(const CouplingParams& p, cudaStream_t s)
{
    if (p.ntasks <= 0) return cudaSuccess;
    if (!p.slices || ((uintptr_t)p.slices & 15u)) return cudaErrorInvalidValue;
    bool n00 = false, n22 = false;
    for (int k = 0; k < p.nwin; ++k) {
        if (p.win[k].product != PROD_22_22) n00 = true;
        if (p.win[k].product != PROD_00_00) n22 = true;
    }
    const uint32_t spec = spec_of(p);
    const Inst* i = find_inst(p, spec);
    return i ? i->launch(p, n00, n22, s) : launch_chosen8(p, spec, n00, n22, s);
}

// Entry j of a window: (2 l3 + 1) W[l3] in FP64, zero for j >= nW, and split.
__device__ __forceinline__ void prep_entry(const double* __restrict__ src, long long nW, int j, double* wW, int2* bf)
{
    const double v = j < nW ? (2.0 * j + 1.0) * src[j] : 0.0;
    wW[j] = v;
    if (bf) bf[j] = split_entry(v);
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
    let_next_start();
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
