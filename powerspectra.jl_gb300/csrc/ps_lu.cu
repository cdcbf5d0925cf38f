// ps_lu.cu -- M \ b in FP64 by LU with partial pivoting, for the matrix sizes of the decoupling step.
//
// The decoupling `M \ pCl` of master (src/modecoupling.jl:358, src/blockspectralmatrix.jl:124-129)
// factors one matrix of a few hundred to a few thousand rows for a few right-hand sides.  At these
// sizes the column-by-column work of the panels bounds a factorisation (cuSOLVER's getrf spends 4.7 us
// per column in its pivoting kernels, 7.4 of 10.6 ms at n = 1532), not the matrix products.
//
// Right-looking, panels of 32 columns; the right-hand sides are further columns, so the forward
// substitution is part of the elimination.  Per panel:
//   * k_lu_panel: one thread-block cluster, four threads per row with the row's 32 values in registers.
//     Per column every block finds its largest entry (warp reductions on the bits of |a|) and sends that
//     row, its key and the pivot's reciprocal to all blocks' shared memory in words that count towards an
//     mbarrier there (bounded wait; a wait that gives up is reported, see below).  So every block knows the pivot row
//     without a cluster barrier (whose memory fence took 0.2 us per column) and eliminates its own rows.  Two sets of
//     buffers alternate: a block sends for column j + 1 only after all of its threads have read column
//     j's, so column j + 2's words meet free buffers.  The kernel leaves the panel's net permutation.
//   * k_lu_rows: a warp per further column applies that permutation and solves with the panel's unit
//     lower triangle (lane = row).
//   * k_lu_update: the FP64 product of the panel's lower part and those rows, in 32 x 32 tiles: small
//     ones, since the FP64 pipe (2 lanes per cycle and SM) gains nothing from larger ones and the last
//     wave stays short.
// The next panel's columns are brought up to date first, on a stream of their own, and the next panel
// runs there while the rest is updated: the panels' chain of barriers (2.3 us per column) and the products
// hide each other.
//
// Back substitution takes one launch per 32 rows: every block solves the diagonal triangle and then
// takes the new values out of its own rows.
//
// The pivot is the entry of largest magnitude, the uppermost one among equals.  A zero pivot is
// reported (info), as getrf does.
//
// When a wait gives up, the panel leaves the rows of the columns beyond it where they are (perm the identity), info
// becomes -1 and the panels after it do nothing, so that everything queued behind stays inside the matrix and ends.
#include "ps_internal.cuh"
#include "ps_umma.cuh"

#include <cooperative_groups.h>

#include <atomic>
#include <limits.h>

namespace cg = cooperative_groups;

namespace ps {
namespace {

constexpr int kPan = 32;          // columns of a panel
constexpr int kMaxCluster = 16;
constexpr int kMaxRows = 256;     // rows per block of the panel kernel, four threads each
constexpr unsigned kNoRow = 0x7fffffffu;

// What a block sends to every block of the cluster for one column: its best row.
struct Cand {
    double row[kPan];             // its columns from the current four on
    double rcp;                   // 1 / pivot
    unsigned long long bits, at;  // of |pivot|; the row's place in the panel
};
constexpr unsigned kCandBytes = sizeof(Cand);
static_assert(kCandBytes == (kPan + 3) * 8, "a candidate is sent in 8-byte words");
struct PanelSmem {
    Cand cand[2][kMaxCluster];
    uint64_t full[2];           // the cluster's candidates have arrived
    double row[kPan];           // this block's candidate before it is sent
    double col[2][kMaxRows];    // a column of this block's rows; two, since a slow warp may still read the last one
    unsigned whi[kMaxRows / 32], wlo[kMaxRows / 32], wat[kMaxRows / 32];  // per 32 rows
    int sent[kMaxCluster];      // columns each block has sent, negative where one of its waits gave up
};

// The largest (hi, lo) of the lanes and the smallest `at` among those that hold it.
__device__ __forceinline__ void best_of(unsigned& hi, unsigned& lo, unsigned& at)
{
    const unsigned h = __reduce_max_sync(0xffffffffu, hi);
    const unsigned l = __reduce_max_sync(0xffffffffu, hi == h ? lo : 0u);
    at = __reduce_min_sync(0xffffffffu, hi == h && lo == l ? at : kNoRow);
    hi = h;
    lo = l;
}
// v to the same place of block d's shared memory, where it counts towards the barrier `full`
__device__ __forceinline__ void send(void* at, uint64_t* full, int d, unsigned long long v)
{
    uint32_t a, m;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(umma::smem_addr(at)), "r"(d));
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(m) : "r"(umma::smem_addr(full)), "r"(d));
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a), "l"(v), "r"(m)
                 : "memory");
}
// Bounded wait of the whole block for phase `parity`, with the other blocks' words visible after it;
// the same answer for every thread.
__device__ __forceinline__ bool wait_full(uint64_t* bar, uint32_t parity, int limit)
{
    const uint32_t a = umma::smem_addr(bar);
    bool done = false;
    for (int it = 0; it < limit && !done; ++it) {
        uint32_t p;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(p)
            : "r"(a), "r"(parity)
            : "memory");
        done = p != 0;
    }
    return __syncthreads_and(done);
}
__device__ __forceinline__ bool is_inf(double x) { return (__double2hiint(x) & 0x7fffffff) == 0x7ff00000 && __double2loint(x) == 0; }

// Panel of w columns from column j0 of the n x n matrix a (leading dimension n).  perm[i], i < 32: the
// row (of those from j0) now at place i; perm[32 + i]: the place of the row that was i, if 32 or beyond,
// else -1.  `rows` rows per block; warp 4 g + q holds the columns q, q + 4, ... of the rows 32 g .. 32 g + 31
// (a warp's FP64 instruction takes 64 cycles of its quarter of an SM: with whole rows in one warp the
// elimination alone took 1000 cycles per column; four quarters share it).  A row stays with its threads;
// a swap exchanges places only, and the finished columns wait in shared memory for the final places.
// The columns run in a loop over four at a time (the registers move up): unrolled over all 32, every
// instruction ran once per panel and its fetch cost more than its work.
// OTHER_LIMIT: the waits give up after `limit` polls, else after kLuWaitLimit (as a number in a register the limit
// costs 1 % of a solve).
template <bool OTHER_LIMIT>
__global__ void __launch_bounds__(4 * kMaxRows, 1) k_lu_panel(double* __restrict__ a, int n, int j0, int w, int rows,
                                                           int* __restrict__ perm, int* info, int limit)
{
    constexpr int kOwn = kPan / 4;  // columns per thread
    extern __shared__ __align__(16) double fin[];  // [column][row of this block, in whole warps]
    __shared__ PanelSmem sm;
    cg::cluster_group cluster = cg::this_cluster();
    const int nb = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    const int q = warp & 3, group = warp >> 2, ngroup = nwarp >> 2, r = 32 * group + lane, nr = 32 * ngroup;
    if (threadIdx.x == 0) {
        umma::mbar_init(&sm.full[0]);
        umma::mbar_init(&sm.full[1]);
    }
    wait_for_previous(j0);  // the update of these columns
    const int m = n - j0;
    auto leave_rows = [&] {  // a panel without a factorisation
        if (rank == 0 && threadIdx.x < kPan) {
            perm[threadIdx.x] = (int)threadIdx.x;
            perm[kPan + threadIdx.x] = -1;
        }
    };
    // set by an earlier panel (this one sets it behind the cluster's last barrier but one): the same for every block
    const int state = *(volatile int*)info;
    const unsigned orig = (unsigned)(rank * rows + r);  // this thread's row
    unsigned at = orig;                                 // and its place
    const bool own = r < rows && orig < (unsigned)m;
    double* A = a + (size_t)j0 * n + j0;
    double v[kOwn];  // v[i]: column q + 4 i from the current four on
#pragma unroll
    for (int i = 0; i < kOwn; ++i) v[i] = own && 4 * i + q < w ? A[(size_t)(4 * i + q) * n + orig] : 0.0;
    if (state < 0) {  // looked at here, its load runs beside the others (ahead of them: 1 us per panel)
        leave_rows();
        return;
    }
    cluster.sync();  // every block's barriers are up before any block writes to its shared memory
    bool ok = true;  // the same for every thread of a block
    int sent = 0;    // columns sent: a block sends one only when it has everyone's of the one before, so that the
                     // blocks' counts differ by one at most
    for (int jq = 0; jq < w; jq += 4) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int j = jq + e;
            if (j < w && ok) {
                const int buf = e & 1;
                const bool mine = q == e, live = own && at >= (unsigned)j;  // mine: this warp holds column j
                // ---- this block's candidate ----
                unsigned hi, lo, row;
                if (mine) {
                    const unsigned long long bits = live ? (unsigned long long)__double_as_longlong(fabs(v[0])) : 0ull;
                    hi = (unsigned)(bits >> 32);
                    lo = (unsigned)bits;
                    row = live ? at : kNoRow;
                    best_of(hi, lo, row);
                    if (lane == 0) {
                        sm.whi[group] = hi;
                        sm.wlo[group] = lo;
                        sm.wat[group] = row;
                    }
                    sm.col[buf][r] = v[0];
                }
                __syncthreads();
                hi = lane < ngroup ? sm.whi[lane] : 0u;
                lo = lane < ngroup ? sm.wlo[lane] : 0u;
                row = lane < ngroup ? sm.wat[lane] : kNoRow;
                best_of(hi, lo, row);
                if (live && at == row) {
                    if (mine) {  // the pivot's reciprocal goes out by itself, while the row is put together
                        const double rcp = hi == 0u && lo == 0u ? 0.0 : 1.0 / v[0];
                        for (int d = 0; d < nb; ++d)
                            send(&sm.cand[buf][rank].rcp, &sm.full[buf], d, (unsigned long long)__double_as_longlong(rcp));
                    }
#pragma unroll
                    for (int i = 0; i < kOwn; ++i) sm.row[4 * i + q] = v[i];
                }
                if (threadIdx.x == 0) umma::mbar_expect_tx(&sm.full[buf], (unsigned)nb * kCandBytes);
                __syncthreads();
                // ---- to every block, a warp per destination ----
                for (int d = warp; d < nb; d += nwarp) {
                    Cand& c = sm.cand[buf][rank];
                    send(&c.row[lane], &sm.full[buf], d, (unsigned long long)__double_as_longlong(sm.row[lane]));
                    if (lane == 0) send(&c.bits, &sm.full[buf], d, (unsigned long long)hi << 32 | lo);
                    if (lane == 1) send(&c.at, &sm.full[buf], d, row);
                    if (lane == 2 && row == kNoRow) send(&c.rcp, &sm.full[buf], d, 0ull);  // no row left here
                }
                sent = j + 1;
                ok = wait_full(&sm.full[buf], (unsigned)(j >> 1) & 1u, OTHER_LIMIT ? limit : kLuWaitLimit);
                if (!ok) continue;  // the candidates are not all here; the columns left are passed over
                // ---- the pivot, the places, the elimination ----
                const unsigned long long kb = lane < nb ? sm.cand[buf][lane].bits : 0ull;
                hi = (unsigned)(kb >> 32);
                lo = (unsigned)kb;
                const unsigned mine_at = lane < nb ? (unsigned)sm.cand[buf][lane].at : kNoRow;
                row = mine_at;
                best_of(hi, lo, row);  // row: the pivot's place, j or below
                const Cand& c = sm.cand[buf][__ffs(__ballot_sync(0xffffffffu, mine_at == row)) - 1];
                if (hi == 0u && lo == 0u && rank == 0 && threadIdx.x == 0) atomicMin(info, j0 + j + 1);
                if (at == row) at = (unsigned)j;
                else if (at == (unsigned)j) at = row;
                if (own && at > (unsigned)j) {
                    // a reciprocal that overflows (a pivot below 2^-1022) gives way to the division
                    const double x = sm.col[buf][r], rcp = c.rcp;
                    const double l = is_inf(rcp) ? x / c.row[e] : x * rcp;
                    if (q > e) v[0] = fma(-l, c.row[q], v[0]);  // the next column first
                    else if (mine) v[0] = l;
#pragma unroll
                    for (int i = 1; i < kOwn; ++i)
                        if (jq + 4 * i < w) v[i] = fma(-l, c.row[4 * i + q], v[i]);
                }
            }
        }
        fin[(jq + q) * nr + r] = v[0];
#pragma unroll
        for (int i = 0; i + 1 < kOwn; ++i) v[i] = v[i + 1];
    }
    // a block that has every column knows its rows' places, whatever becomes of the others
    if (own && ok) {
#pragma unroll
        for (int i = 0; i < kOwn; ++i)
            if (4 * i + q < w) A[(size_t)(4 * i + q) * n + at] = fin[(4 * i + q) * nr + r];
        if (q == 0) {  // row `orig` is at place `at` now
            if (at < (unsigned)kPan) perm[at] = (int)orig;
            if (orig < (unsigned)kPan) perm[kPan + orig] = at < (unsigned)kPan ? -1 : (int)at;
        }
    }
    // ---- the end, for all blocks alike ----
    if (threadIdx.x < nb) *cluster.map_shared_rank(&sm.sent[rank], (int)threadIdx.x) = ok ? sent : -sent;
    cluster.sync();  // no block leaves while another may write to it
    int top = 0;
    bool all = true;
    for (int b = 0; b < nb; ++b) {
        top = max(top, abs(sm.sent[b]));
        all &= sm.sent[b] > 0;
    }
    if (!all) {
        // No block may leave while words are under way to it.  Those of the last column, top - 1, come from the
        // blocks that sent it; the others send words without a meaning, so that it completes everywhere.
        if (sent < top) {
            uint64_t* full = &sm.full[(top - 1) & 1];
            Cand& c = sm.cand[(top - 1) & 1][rank];
            if (threadIdx.x == 0) umma::mbar_expect_tx(full, (unsigned)nb * kCandBytes);
            for (int e = threadIdx.x; e < nb * (kPan + 3); e += blockDim.x)
                send(&c.row[0] + e % (kPan + 3), full, e / (kPan + 3), 0ull);
        }
        for (int j = max(top - 2, 0); j < top; ++j) wait_full(&sm.full[j & 1], (unsigned)(j >> 1) & 1u, kLuWaitLimit);
        leave_rows();
        if (threadIdx.x == 0) atomicMin(info, -1);
        cluster.sync();
    }
}

// The columns cb .. ce - 1 beyond the panel: rows permuted, then the first w of them solved with the
// panel's unit lower triangle.  A warp per column, lane = row.  Columns n and beyond are those of b.
__global__ void __launch_bounds__(256) k_lu_rows(double* __restrict__ a, double* __restrict__ b, int n, int cb, int ce,
                                                 int j0, int w, const int* __restrict__ perm)
{
    __shared__ double L[kPan][kPan + 1];  // [column][row]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    let_next_start();
    for (int k = warp; k < kPan; k += 8)
        L[k][lane] = k < lane && lane < w ? a[(size_t)(j0 + k) * n + j0 + lane] : 0.0;
    __syncthreads();
    const int c = cb + blockIdx.x * 8 + warp;
    if (c >= ce) return;
    double* col = (c < n ? a + (size_t)c * n : b + (size_t)(c - n) * n) + j0;
    const int m = n - j0;
    const bool in = lane < kPan && lane < m;  // with fewer than 32 rows left all are in the panel
    const int from = in ? perm[lane] : 0, to = in ? perm[kPan + lane] : -1;
    double x = in ? col[from] : 0.0;
    const double y = in ? col[lane] : 0.0;
    __syncwarp();
    if (lane >= w) x = 0.0;
#pragma unroll
    for (int k = 0; k + 1 < kPan; ++k)  // L is 0 beyond the panel and, as read here, from the diagonal up
        x = fma(-L[k][lane], __shfl_sync(0xffffffffu, x, k), x);
    if (in) col[lane] = x;
    if (to >= 0) col[to] = y;
}

// a[i, c] -= sum_k L[i, k] U[k, c] for the rows i >= j0 + 32 and the columns c = cb .. ce - 1 (b's too)
__global__ void __launch_bounds__(128) k_lu_update(double* __restrict__ a, double* __restrict__ b, int n, int cb,
                                                   int ce, int j0)
{
    __shared__ __align__(16) double L[kPan][32], U[kPan][32 + 2];  // L[k][row], U[k][column]
    int i0 = j0 + kPan + blockIdx.x * 32;
    const int c0 = cb + blockIdx.y * 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    let_next_start();
    for (int k = warp; k < kPan; k += 4) L[k][lane] = i0 + lane < n ? a[(size_t)(j0 + k) * n + i0 + lane] : 0.0;
    wait_for_previous(j0, i0);  // the rows of U (the panel itself was complete before that kernel)
    for (int q = warp; q < 32; q += 4) {
        const int c = c0 + q;
        U[lane][q] = c < ce ? (c < n ? a + (size_t)c * n : b + (size_t)(c - n) * n)[j0 + lane] : 0.0;
    }
    __syncthreads();
    // thread: rows 2 tx, 2 tx + 1, columns 4 ty .. 4 ty + 3
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double s[4][2] = {};
#pragma unroll 8
    for (int k = 0; k < kPan; ++k) {
        const double2 l = *reinterpret_cast<const double2*>(&L[k][2 * tx]);
        const double2 u0 = *reinterpret_cast<const double2*>(&U[k][4 * ty]);
        const double2 u1 = *reinterpret_cast<const double2*>(&U[k][4 * ty + 2]);
        const double u[4] = {u0.x, u0.y, u1.x, u1.y};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            s[q][0] = fma(l.x, u[q], s[q][0]);
            s[q][1] = fma(l.y, u[q], s[q][1]);
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int c = c0 + 4 * ty + q;
        if (c < ce) {
            double* col = c < n ? a + (size_t)c * n : b + (size_t)(c - n) * n;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int i = i0 + 2 * tx + e;
                if (i < n) col[i] -= s[q][e];
            }
        }
    }
}

// One step of the back substitution for right-hand side blockIdx.y: its w rows from j0 into x, and their
// contribution out of the rows above (each block its own 256).
__global__ void __launch_bounds__(256) k_lu_back(const double* __restrict__ a, double* __restrict__ b,
                                                 double* __restrict__ x, int n, int j0, int w)
{
    __shared__ double U[kPan][kPan + 1];  // [column][row]
    __shared__ double sx[kPan];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int i = blockIdx.x * 256 + threadIdx.x;
    let_next_start();
    b += (size_t)blockIdx.y * n;
    // what the steps before do not change: the triangle and this thread's row
    for (int k = warp; k < kPan; k += 8)
        U[k][lane] = k < w && lane < w ? a[(size_t)(j0 + k) * n + j0 + lane] : 0.0;
    double v[kPan];
#pragma unroll
    for (int k = 0; k < kPan; ++k) v[k] = i < j0 && k < w ? a[(size_t)(j0 + k) * n + i] : 0.0;
    wait_for_previous(j0, i);
    __syncthreads();
    if (warp == 0) {
        const double r = lane < w ? 1.0 / U[lane][lane] : 0.0;
        const bool divide = __any_sync(0xffffffffu, is_inf(r));  // a diagonal entry below 2^-1022
        double y = lane < w ? b[j0 + lane] : 0.0;
        for (int k = w - 1; k >= 0; --k) {
            const double u = __shfl_sync(0xffffffffu, divide ? y / U[k][k] : y * r, k);
            if (lane == k) y = u;
            if (lane < k) y = fma(-U[k][lane], u, y);
        }
        sx[lane] = y;
        if (blockIdx.x == 0 && lane < w) x[(size_t)blockIdx.y * n + j0 + lane] = y;
    }
    __syncthreads();
    if (i >= j0) return;
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int k = 0; k < kPan; k += 2) {  // v and sx are 0 beyond w
        s0 = fma(v[k], sx[k], s0);
        s1 = fma(v[k + 1], sx[k + 1], s1);
    }
    b[i] -= s0 + s1;
}

constexpr size_t panel_smem(int rows) { return (size_t)kPan * 32 * ((rows + 31) / 32) * sizeof(double); }

cudaLaunchConfig_t panel_config(int blocks, int rows, cudaLaunchAttribute (&at)[2])
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)(128 * ((rows + 31) / 32)));
    cfg.dynamicSmemBytes = panel_smem(rows);
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)blocks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // see launch_after
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cfg;
}

// Most blocks per cluster of the panel kernel on the current device: 16 where it takes such a cluster,
// else 8 (0: none).  Asked once per device.
int cluster_blocks()
{
    constexpr int kMaxDevices = 64;
    static std::atomic<int> known[kMaxDevices];  // blocks + 1; 0: not asked yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        cudaGetLastError();
        return 0;
    }
    if (const int b = known[dev].load()) return b - 1;
    int blocks = 0;
    bool ready = true;
    for (auto kernel : {k_lu_panel<false>, k_lu_panel<true>})
        ready = ready &&
                cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)panel_smem(kMaxRows)) ==
                    cudaSuccess &&
                cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    if (ready)
        for (int b = kMaxCluster; b >= 8 && !blocks; b /= 2) {
            cudaLaunchAttribute at[2];
            const cudaLaunchConfig_t cfg = panel_config(b, kMaxRows, at);
            int nc = 0;
            if (cudaOccupancyMaxActiveClusters(&nc, k_lu_panel<false>, &cfg) == cudaSuccess && nc > 0) blocks = b;
        }
    cudaGetLastError();
    known[dev].store(blocks + 1);
    return blocks;
}

}  // namespace

// Beyond 4096 rows a panel does not fit the cluster's threads, and for many right-hand sides a solve is
// mostly products: cuSOLVER takes those.  Measured as host calls with one right-hand side, cuSOLVER and
// this: n = 96 0.36 and 0.27 ms, n = 400 1.97 and 1.04, n = 1532 11.5 and 5.7, n = 4000 67 and 44.
bool lu_fits(int n, int nrhs) { return nrhs <= 32 && n <= cluster_blocks() * kMaxRows; }

// x = a^-1 b for the n x n device matrix a and nrhs columns b (leading dimensions n), on stream s with the
// panels on w.side; a and b are overwritten.  *w.info becomes the first zero pivot's index from 1, -1 when a
// wait gave up (x then holds nothing of use), or stays INT_MAX.  *launches grows by the kernels launched.
cudaError_t launch_lu_solve(double* a, int n, double* b, int nrhs, double* x, const LuWork& wk, cudaStream_t s, int* launches)
{
    static const int kNone = INT_MAX;
#define LU_TRY(call) \
    if (cudaError_t e_ = (call)) return e_
    LU_TRY(cudaMemcpyAsync(wk.info, &kNone, sizeof(int), cudaMemcpyHostToDevice, s));
    LU_TRY(cudaEventRecord(wk.rest, s));
    LU_TRY(cudaStreamWaitEvent(wk.side, wk.rest, 0));
    const int nb = cluster_blocks(), ncol = n + nrhs;
    auto beyond = [&](int cb, int ce, int j0, int w, const int* perm, cudaStream_t st) -> cudaError_t {
        if (cb >= ce) return cudaSuccess;
        ++*launches;
        k_lu_rows<<<(unsigned)((ce - cb + 7) / 8), 256, 0, st>>>(a, b, n, cb, ce, j0, w, perm);
        const int below = n - j0 - kPan;
        if (below > 0) {
            ++*launches;
            const dim3 grid((unsigned)((below + 31) / 32), (unsigned)((ce - cb + 31) / 32));
            // the next panel's columns are waited for; the rest has time, and its blocks would take their places
            if (st == wk.side) return launch_after(k_lu_update, grid, dim3(128), 0, st, a, b, n, cb, ce, j0);
            k_lu_update<<<grid, 128, 0, st>>>(a, b, n, cb, ce, j0);
        }
        return cudaGetLastError();
    };
    for (int j0 = 0; j0 < n; j0 += kPan) {
        const int w = n - j0 < kPan ? n - j0 : kPan, m = n - j0;
        int* perm = wk.perm + (j0 / kPan & 1) * 2 * kPan;  // the rest of this panel may run beside the next one
        // a cluster of 8 has the quicker barrier, 16 the shorter elimination: even at about 1000 rows
        const int blocks = nb > 8 && m > 1024 ? nb : 8, rows = (m + blocks - 1) / blocks;
        cudaLaunchAttribute at[2];
        cudaLaunchConfig_t cfg = panel_config(blocks, rows, at);
        cfg.stream = wk.side;
        if (j0 == 0) cfg.numAttrs = 1;  // the first one has no update before it
        const auto kernel = wk.wait_limit == kLuWaitLimit ? k_lu_panel<false> : k_lu_panel<true>;
        ++*launches;
        LU_TRY(cudaLaunchKernelEx(&cfg, kernel, a, n, j0, w, rows, perm, wk.info, wk.wait_limit));
        LU_TRY(cudaEventRecord(wk.panel, wk.side));
        LU_TRY(cudaStreamWaitEvent(s, wk.panel, 0));
        const int c1 = j0 + w, c2 = c1 + kPan < n ? c1 + kPan : (n > c1 ? n : c1);  // the next panel: c1 .. c2 - 1
        if (c1 < c2 && j0 > 0) LU_TRY(cudaStreamWaitEvent(wk.side, wk.rest, 0));
        LU_TRY(beyond(c1, c2, j0, w, perm, wk.side));
        LU_TRY(beyond(c2, ncol, j0, w, perm, s));
        LU_TRY(cudaEventRecord(wk.rest, s));
    }
    for (int j0 = (n - 1) / kPan * kPan; j0 >= 0; j0 -= kPan) {
        const int w = n - j0 < kPan ? n - j0 : kPan;
        const dim3 grid((unsigned)(j0 > 0 ? (j0 + 255) / 256 : 1), (unsigned)nrhs);
        ++*launches;
        if (j0 + kPan >= n) {  // the first one starts when the matrix is done
            k_lu_back<<<grid, 256, 0, s>>>(a, b, x, n, j0, w);
            LU_TRY(cudaGetLastError());
        } else {
            LU_TRY(launch_after(k_lu_back, grid, dim3(256), 0, s, a, b, x, n, j0, w));
        }
    }
#undef LU_TRY
    return cudaSuccess;
}

}  // namespace ps
