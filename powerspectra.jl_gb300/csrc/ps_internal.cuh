// ps_internal.cuh -- shared declarations of the powerspectra_gpu library.
//
// Data layout on the device (one context owns all of it, reused across calls):
//   * windows:  K padded rows of length wlen = 2*lmax + 2 holding
//               (2 l3 + 1) * W_k[l3] for l3 < nW and 0 beyond, so every family
//               read (l3 <= l1 + l2 <= 2 lmax) stays in bounds without a branch.
//   * tasks:    int2 (l1, l2_0) per warp, 32 consecutive l2 of one l1 row,
//               heaviest rows first (the family length is 2 l1 + 1), tiled:
//               kTileRows consecutive rows per block over one 32-column block
//               (see tile_task_list in ps_api.cu).
//   * half:     the plain kernels' table of C(n), 1 / (C(n) (n + 1)) and
//               2 pi (2 j + 1) (HalfTable), kept per context.
//   * outputs:  column-major (Julia) matrices, element (l1, l2) at
//               (l1 - lmin) + (l2 - lmin) * ld.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>

#include "../../include/powerspectra_gpu.h"

namespace ps {

constexpr int kMaxWin = 8;       // windows (slots) per coupling launch
constexpr int kWarpsPerBlock = 4;
constexpr int kTileRows = 4;  // rows per tile of the task list (one per warp)
constexpr double kInv4Pi = 0.079577471545947667884;  // 1 / (4 pi)

// Family product a window is contracted with.
enum Product : int { PROD_00_00 = 0, PROD_22_22 = 1, PROD_00_22 = 2 };
// l3 parity filter relative to l1 + l2 + l3.
enum Parity : int { PAR_ALL = 0, PAR_EVEN = 1, PAR_ODD = 2 };
// What the kernel writes per pair.
enum Epilogue : int { EPI_MCM = 0, EPI_XI = 1, EPI_COV = 2 };

struct WinDesc {
    const double* wW;  // padded (2 l3 + 1) W[l3], length wlen >= 2 lmax + 2
    const int2* bf;    // the same values split as (float mantissa bits, int exponent): what slices are made of
    int product;
    int parity;
};

// The factors of the squared (0 0 0) symbol (ps_plain_fp64.cu), for lmax: C[n] = Gamma((n + 1) / 2) /
// (sqrt(pi) Gamma(n / 2 + 1)) and U[n] = 1 / (C[n] (n + 1)) for n = 0 .. top, and W[j] = 2 pi (2 j + 1)
// for j = 0 .. 2 lmax + 1.
struct HalfTable {
    const double *C, *U, *W;
    int top;
};

// A kernel launched by launch_after starts while the one before it in the stream still runs (once all of that
// one's blocks have called let_next_start or ended), so its launch and the start of its blocks cost no time of
// their own: TT at lmax 767 104.6 -> 96.8 us, the chain of short kernels of a 1532-row solve 6.32 -> 5.73 ms.
// Not worth it beside kernels that fill the memory system (window spectra at lmax 2508 78.5 -> 84.9 us) nor
// where a long kernel's addresses take the detour (tensor-core kernels at lmax 8191 424.5 -> 428.8 ms).  All of its threads call wait_for_previous before anything that the kernel
// before it writes or reads; what came earlier in the stream is complete.  x: a value on which
// the addresses of every load of such data depend (loads through the read-only path are otherwise free to move up).
#ifdef __CUDACC__
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous(int& x) { asm volatile("griddepcontrol.wait;" : "+r"(x)::"memory"); }
__device__ __forceinline__ void wait_for_previous(int& x, int& y)
{
    asm volatile("griddepcontrol.wait;" : "+r"(x), "+r"(y)::"memory");
}
constexpr unsigned kSMs = 152;
// Dynamic shared memory with which at most `blocks` blocks of a kernel with `fixed` bytes share an SM (228 KB,
// 1 KB of it per block).
constexpr size_t kSmemSM = 228 * 1024;
constexpr size_t pad_smem(int blocks, size_t fixed)
{
    const size_t need = kSmemSM / (blocks + 1) / 128 * 128 + 128, have = 1024 + fixed;
    return need > have ? need - have : 0;
}
// Lets a kernel be launched with `bytes` of dynamic shared memory.  The limit set is the same for every launch, so
// that of one thread never undercuts another's (with 48 KB of static memory it stays within a block's 227 KB).
constexpr size_t kDynLimit = 160 * 1024;
template <class K>
inline cudaError_t allow_smem(K kernel, size_t bytes)
{
    return bytes ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDynLimit) : cudaSuccess;
}
static_assert(pad_smem(1, 0) <= kDynLimit, "one block per SM is the largest pad");
template <class... P, class... A>
inline cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args)
{
    if (cudaError_t e = allow_smem(kernel, smem)) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
#endif

// The square-root ratios of the chosen kernels' recurrences (chosen_xi), float-float pairs (rho, r) of 16
// bytes, for every row l1 <= lmax.  With F(a) = a (a + 2 l1 + 1) and G(t) = t (2 l1 + 1 - t):
//   f, entry a:  -sqrt(F(a) / F(a + 1)), 1 / sqrt(F(a + 1))   a = -62 .. 2 lmax - l1 + 94, zeros below a = 0
//   b, entry a:  -sqrt(F(a + 1) / F(a)), 1 / sqrt(F(a))       a = l1 - 92 .. 2 lmax + 64, zeros up to a = 0
//   g, entry t:   sqrt(G(t) / G(t + 1)), 1 / sqrt(G(t + 1))   t = 0 .. l1 - 1
struct CoefRows {
    const float4 *f, *b, *g;  // f null: no table
    int lmax;                 // of the table: at least that of the launches that read it
};
__host__ __device__ constexpr long long coef_row(int lmax, int l1)  // first entry of row l1 in f and b
{
    return (long long)l1 * (2 * lmax + 160) - (long long)l1 * (l1 - 1) / 2;
}
__host__ __device__ constexpr long long coef_row_g(int l1) { return (long long)l1 * (l1 - 1) / 2; }
// rows 0 .. lmax of f, then of b, then of g (a warp reads 32 entries at a time, past the last row's end)
constexpr size_t coef_bytes(int lmax)
{
    return (size_t)(2 * coef_row(lmax, lmax + 1) + coef_row_g(lmax + 1) + 32) * sizeof(float4);
}
inline CoefRows coef_rows(const float4* t, int lmax)
{
    const long long n = coef_row(lmax, lmax + 1);
    return CoefRows{t, t + n, t + 2 * n, lmax};
}

struct CouplingParams {
    int lmin, lmax;
    int nwin;
    WinDesc win[kMaxWin];
    const int2* tasks;
    int ntasks;
    int epilogue;
    double* out[kMaxWin];  // EPI_MCM / EPI_XI: one matrix per window; EPI_COV: out[0]
    long long ldo;
    int wlen;  // length of the padded window arrays
    int nw;    // their entries at l3 >= nw are zero
    // chosen kernel: the windows themselves (device pointers, nw entries), for launches that prepare the
    // rows win[k].wW with their slices and leave win[k].bf unset; src[0] null otherwise
    const double* src[kMaxWin];
    int cov_kind;
    const double* S[4];  // covariance signal spectra (length >= lmax + 1), reference argument order
    const double* R[4];  // covariance noise ratios
    HalfTable half;      // the plain kernel's factors (unset for the chosen kernel)
    unsigned char* slices;  // the chosen kernel's table of window slices (slice_table_bytes of scratch)
    CoefRows coef;          // the chosen kernel's square-root ratios, or none (it makes them itself)
};

// One window of a batch: user spectrum -> padded (2l+1)W row and its split copy.
struct WinPrep {
    const double* src;
    long long nW;
    double* wW;
    int2* bf;
    int wlen;
};

// Persistent batched launch: groups[item.x] holds the coupling parameters of
// an item int4 (group, l1, first l2, w) with w = tasks | families << 8 |
// kernel body << 12 (families: 1 = 00 only, 2 = 22 only, 3 = both).
struct BatchParams {
    const CouplingParams* groups;
    const int4* items;
    int nitems;
    bool coef;  // the groups have a table of square-root ratios
    unsigned* counter;  // work-queue head, zeroed before every launch
};

// Launchers (ps_plain_fp64.cu, ps_chosen.cu).
// The batched kernel with NWIN = 4 or 8 slots per group (nwin > 4 selects 8).
cudaError_t launch_batch_chosen(const BatchParams& bp, int blocks, int nwin, cudaStream_t s);
int batch_blocks_per_sm(int nwin, bool coef);  // of the kernel that launch_batch_chosen takes
int chosen_batch_template(const CouplingParams& p, int nwin);  // compile-time slot set of a batch group (0: none fits)
cudaError_t launch_prep_windows(const WinPrep* list, int n, int max_wlen, cudaStream_t s);
cudaError_t launch_plain_fp64(const CouplingParams& p, cudaStream_t s);
// Two launches: the table of window slices into p.slices (16-byte aligned), then the coupling kernel.
cudaError_t launch_chosen(const CouplingParams& p, cudaStream_t s);
size_t slice_table_bytes(const CouplingParams& p);
size_t slice_table_most(int lmax);  // for any list of slots
// The table of square-root ratios (coef_bytes(lmax)), and whether launch_chosen reads one if p.coef has it.
cudaError_t launch_coef(float4* t, int lmax, cudaStream_t s);
bool reads_coef(const CouplingParams& p);
bool has_coef(const CouplingParams& p);  // ... at any lmax
// Smaller lmax in a batch: no table, each warp makes its few slices itself.  Then a table holds more slices than are
// read, and its kernel comes on top.  Without and with tables, n x lmax, all spins: 2000 x 32 516 and 607 us, 300 x 100 612
// and 629, 200 x 127 660 and 662, 100 x 250 1496 and 1420.  The (0 0 0) family alone has half the steps: one window 4 x 200 93 and
// 101, 100 x 250 777 and 779, 1 x 500 279 and 260; four windows 100 x 160 334 and 337, 4 x 200 100 and 92; eight 100 x 160 776 and 694.
inline int slice_min_lmax(const CouplingParams& g)
{
    for (int k = 0; k < g.nwin; ++k)
        if (g.win[k].product != PROD_00_00) return 128;
    return g.nwin > 4 ? 128 : (g.nwin > 2 ? 192 : 300);
}
// The slice tables of a batch's groups (NWIN = 4 or 8 as for launch_batch_chosen), each into its group's own p.slices
// of batch_slice_bytes(lmax, nwin): block b makes kSliceBlock entries of group blocks[b].x, from entry blocks[b].y &
// 0xffffff of slice_entries(lmax), of window blocks[b].y >> 24.
constexpr int kSliceBlock = 64;
cudaError_t launch_batch_slices(const CouplingParams* groups, const int2* blocks, int nblocks, int nwin, cudaStream_t s);
int slice_entries(int lmax);
size_t batch_slice_bytes(int lmax, int nwin);
// K windows of nW entries (device pointers in a host array) into padded rows wW + k wlen of (2l+1) W[l]
// and, when bf is given, their split copies bf + k wlen, one launch per kSetWindows windows.
constexpr int kSetWindows = 64;
inline int set_launches(int K) { return (K + kSetWindows - 1) / kSetWindows; }
cudaError_t launch_prep_set(const double* const* src, int K, long long nW, int wlen, double* wW, int2* bf,
                            cudaStream_t s);

// Exponent marking an exact zero in the split window arrays.
constexpr int kZeroExp = -100000;
cudaError_t launch_fma_probe(int fp64, double* sink, int blocks, int iters, cudaStream_t s);
// LU solve of the decoupling step (ps_lu.cu).
bool lu_fits(int n, int nrhs);
struct LuWork {
    cudaStream_t side;         // the panels' stream
    cudaEvent_t panel, rest;
    int* perm;                 // 128 ints
    int* info;
    int wait_limit;            // polls of a panel's waits
};
constexpr int kLuWaitLimit = 1 << 22;
cudaError_t launch_lu_solve(double* a, int n, double* b, int nrhs, double* x, const LuWork& wk, cudaStream_t s,
                            int* launches);
cudaError_t launch_transpose(double* dst, const double* src, int n, cudaStream_t s);
cudaError_t launch_negate(double* a, long long count, cudaStream_t s);
// scratch: quickpol_scratch(lmax) doubles; half: for lmax
size_t quickpol_scratch(int lmax);
cudaError_t launch_quickpol(const double* W, long long nW, int lmax, int bl, int bu, int nu1, int nu2, int s1, int s2,
                            double* Xi, long long ldx, const HalfTable& half, double* scratch, cudaStream_t s);
// The chosen-arithmetic QuickPol Xi (ps_quickpol_ff.cu); wf: nW floats, e: one int of scratch.
cudaError_t launch_quickpol_ff(const double* W, long long nW, int lmax, int bl, int bu, int nu1, int nu2, int s1,
                               int s2, double* Xi, long long ldx, float* wf, int* e, cudaStream_t s);

// alm2cl reduction (ps_window.cu).  Term t pairs coefficient sets a[t], b[t]
// (HEALPix m-major order, lmax / mmax); a null set stands for all zeros.
constexpr int kAlmMaxTerms = 16;
constexpr int kAlmChunk = 64;  // most m values per block of the partial-sum kernel
struct AlmParams {
    const double2* a[kAlmMaxTerms];
    const double2* b[kAlmMaxTerms];
    int nterms;
    int lmax, mmax, lout;
    int mchunk, nmchunks;
    double* partial;  // nterms * nmchunks * (lout + 1)
};
int alm2cl_chunk(int mmax, int lout);  // m values per chunk
size_t alm2cl_partials(int mmax, int lout);  // room for a term's partial sums
// after_partial, when given, is recorded between the partial-sum kernel and the reduction.
cudaError_t launch_alm2cl(const AlmParams& p, double scale, bool per_l, double* W, cudaStream_t s,
                          cudaEvent_t after_partial = nullptr);

// Tensor-core coupling kernels for sets of windows (ps_mma.cu): up to
// kMmaMaxSlots windows per launch, all with the squared (2 -2 0) family (each
// with a parity) or all with the squared (0 0 0) family (PAR_ALL), contracted
// on the tensor cores; one more MMA column forms the normalisation.
constexpr int kMmaCols = 16;
constexpr int kMmaMaxSlots = kMmaCols - 1;
struct MmaParams {
    int lmin, lmax;
    int nslot;                          // 1 .. kMmaMaxSlots
    const int2* bf[kMmaMaxSlots];       // split windows (mantissa, exponent), length wlen
    const double* wW[kMmaMaxSlots];     // padded windows (2 l3 + 1) W[l3]: the last forward point in FP64
    int parity[kMmaMaxSlots];           // PAR_ALL / PAR_EVEN / PAR_ODD of l1 + l2 + l3
    double* out[kMmaMaxSlots];
    long long ldo;
    int wlen;
    int epilogue;                       // EPI_MCM or EPI_XI
    int stage_rows;                     // 1: outputs in host memory, their scattered half staged
    const int2* tiles;                  // (r0, c0): rows r0 + 2w, columns c0 + 2i
    int ntiles;
    unsigned* status;                   // set to 1 when a bounded wait gives up
    // scratch of mma_table_bytes(lmax) bytes (256-byte aligned) for the launch's table of B
    // tiles; launch_mma fills it, and the entry ranges below, on the stream before the kernel
    unsigned char* tab;
    int tab_fmin, tab_nf, tab_bmin, tab_nb;  // forward entries l3 = fmin .. fmin + nf - 1, then backward ones
};
// fam00: the (0 0 0) family (every slot PAR_ALL); otherwise the (2 -2 0) family.  Two
// launches: the table of B tiles, then the coupling kernel.
cudaError_t launch_mma(const MmaParams& p, bool fam00, cudaStream_t s);
size_t mma_table_bytes(int lmax);

// A covariance block from its Xi matrices (ps_cov_combine.cu): C[l1, l2] =
// cov_combine(kind, S, R, {X_k[l1, l2]}, l1, l2) over the whole n x n block.
struct CovCombineParams {
    int kind, lmin, n, nx;     // nx: the block's windows (cov_nwindows(kind))
    const double* S[4];
    const double* R[4];
    const double* X[kMaxWin];  // the block's windows' Xi, n x n, leading dimension ldx
    long long ldx;
    double* C;
    long long ldc;
};
cudaError_t launch_cov_combine(const CovCombineParams& p, cudaStream_t s);

// Host-side covariance table (ps_api.cu).
int cov_nwindows(int kind);
int cov_nratios(int kind);
void cov_window_spec(int kind, int k, int* product, int* parity);

}  // namespace ps
