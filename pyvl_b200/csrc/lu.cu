// Dense FP64 LU with partial pivoting (GEPP) and the matching solve, for the row-major
// system matrix the induction kernels write.  Replaces the reference's
// scipy.linalg.lu_factor / lu_solve (python/pyvl/solver.py:223-227).
//
// Right-looking blocked factorisation, panel width NB = 64, one panel of look-ahead.  Per panel:
//   1. the diagonal block and its inverses, and 2. the multipliers and the row block, as if no
//      row interchange were needed (lu_panel.cuh), each fused with the previous panel's update;
//   3. panel_pivot_kernel -- if partial pivoting would have chosen other rows (some multiplier
//      not below 1 in magnitude), the panel is restored from its backup and factored with
//      explicit partial pivoting in getf2 order;
//   4. trsm_kernel -- that panel's interchanges applied to the other columns and its
//      U12 = L11^-1 A12 by substitution (nothing to do for an accepted panel);
//   5. dmma_update_kernel -- A22 -= L21 U12 beyond the next panel, on a side stream beside the
//      next panel's steps 1 and 2.
// Diagonally dominant systems (the vortex-ring matrices are close to -2 pi I) are accepted on
// every panel; a bordered closed-body system falls back on the panel holding the zero-diagonal
// border.  The FP32 factorisation below keeps its own panel kernel (panel_spec_kernel).
//
// The solve runs two wavefront kernels (trsv.cuh; forward with unit-lower L, backward with U) over
// row blocks, one CTA per block, co-resident through a cooperative launch; every wait on an
// earlier block is bounded and reports a time-out through a device error word.
#include <algorithm>
#include <cstdint>

#include "pvl_common.cuh"
#include "dmma.cuh"
#include "lu_panel.cuh"
#include "trsv.cuh"

namespace {

constexpr int NB = 64;               // panel width
constexpr int kSlabRows = 64;        // rows below the top block per CTA in panel_spec_kernel
constexpr int kRB = 64;              // rows per block in the wavefront solves
static_assert(kRB == pvl::trsv::kRB, "the solve's row blocks are the inverted diagonal blocks");
static_assert(NB == pvl::dmma::K && NB == pvl::panel::NB, "the tensor-core products have K = the panel width");
constexpr int kSolveThreads = pvl::trsv::kThreads;

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
inline unsigned blocks_for(size_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

struct LuWs {
    double* backup;         // (n, NB) copy of the current panel before speculation
    double* top_out;        // (NB, NB) speculative top block (FP32 path only)
    int32_t* reject;        // per panel: the speculation failed
    int32_t* ok;            // per panel: speculative factors accepted
    double* tmp;            // (n) vector of the blocked solve
    double* inv;            // (n_blocks, 2, kRB, kRB): inverses of the diagonal blocks of L and U
    double* backup_row;     // (NB, n) copy of the panel's row block right of it (FP64 path)
    double* even;           // (n, even_stride(n)) for odd n: the matrix with 128-byte rows (FP64 path)
};

// Row stride of LuWs::even, 0 where the matrix is factored in place.
uint32_t even_stride(uint32_t n) { return n % 2 ? (n + 15) & ~15u : 0; }

// lu32: the FP32 factorisation's, which has no copy of the matrix.
size_t lu_ws_bytes(uint32_t n, bool lu32 = false)
{
    return align256((size_t)n * NB * sizeof(double)) + align256((size_t)NB * NB * sizeof(double)) +
           align256(((size_t)n / NB + 2) * sizeof(int32_t)) +
           align256(((size_t)n / NB + 2) * sizeof(int32_t)) +
           align256((size_t)n * sizeof(double)) + align256(((size_t)n + kRB - 1) / kRB * 2 * kRB * kRB * sizeof(double)) +
           align256((size_t)NB * n * sizeof(double)) +
           (lu32 ? 0 : align256((size_t)n * even_stride(n) * sizeof(double)));
}

LuWs carve(void* ws, uint32_t n)
{
    char* p = static_cast<char*>(ws);
    LuWs w;
    w.backup = reinterpret_cast<double*>(p);
    p += align256((size_t)n * NB * sizeof(double));
    w.top_out = reinterpret_cast<double*>(p);
    p += align256((size_t)NB * NB * sizeof(double));
    w.reject = reinterpret_cast<int32_t*>(p);
    p += align256(((size_t)n / NB + 2) * sizeof(int32_t));
    w.ok = reinterpret_cast<int32_t*>(p);
    p += align256(((size_t)n / NB + 2) * sizeof(int32_t));
    w.tmp = reinterpret_cast<double*>(p);
    p += align256((size_t)n * sizeof(double));
    w.inv = reinterpret_cast<double*>(p);
    p += align256(((size_t)n + kRB - 1) / kRB * 2 * kRB * kRB * sizeof(double));
    w.backup_row = reinterpret_cast<double*>(p);
    p += align256((size_t)NB * n * sizeof(double));
    w.even = reinterpret_cast<double*>(p);
    return w;
}

__global__ void init_perm_kernel(uint32_t n, int32_t* __restrict__ perm)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        perm[i] = (int32_t)i;
}

// dst (row stride ldd) = src (row stride lds), n x n.
__global__ void __launch_bounds__(256) copy_matrix_kernel(uint32_t n, const double* __restrict__ src, uint32_t lds,
                                                          double* __restrict__ dst, uint32_t ldd)
{
    const uint32_t c = blockIdx.x * 256 + threadIdx.x;
    if (c >= n)
        return;
    for (uint32_t r = blockIdx.y; r < n; r += gridDim.y)
        dst[(size_t)r * ldd + c] = src[(size_t)r * lds + c];
}

// ---------------------------------------------------------------- 1+2. speculative panel
// grid.x = max(1, ceil(below / kSlabRows)); 128 threads: threads 0..63 hold the 64 rows of
// the top block (every CTA factors the same top block, so no CTA waits for another), threads
// 64..127 hold this CTA's rows below it.  Each thread keeps its row in registers (columns
// beyond nb are zero; missing top rows are unit rows) and eliminates column j with the row
// that thread j publishes in shared memory, scaling by the reciprocal of the pivot as getf2
// does -- the recurrence of getf2 without interchanges.  Partial pivoting would keep the
// diagonal in column j iff no entry below it is larger in magnitude at that moment; every
// thread checks this for its own row, and any violation (or a zero/NaN pivot) marks the panel.
// Slab rows are backed up and overwritten in place; the factored top block goes to `top_out`
// (committed by panel_pivot_kernel) so that no CTA can read a half-written top block.
template <typename T>
__global__ void __launch_bounds__(2 * kSlabRows) panel_spec_kernel(uint32_t n, uint32_t k0, uint32_t nb,
                                                                   T* __restrict__ A, uint32_t lda,
                                                                   T* __restrict__ backup,
                                                                   T* __restrict__ top_out,
                                                                   int32_t* __restrict__ reject)
{
    __shared__ T U[NB][NB + 1];
    __shared__ T s_rcp[NB];
    const uint32_t tid = threadIdx.x;
    const bool is_top = tid < NB;
    const uint32_t r_begin = k0 + nb + blockIdx.x * kSlabRows;
    // global row of this thread (top: k0 + tid, slab: r_begin + tid - 64)
    const uint32_t grow = is_top ? k0 + tid : r_begin + (tid - NB);
    const bool valid = is_top ? tid < nb : grow < n;
    T row[NB];
#pragma unroll
    for (int c = 0; c < NB; ++c) {
        T v = T(0);
        if (valid && (uint32_t)c < nb)
            v = A[(size_t)grow * lda + k0 + c];
        else if (is_top && !valid && (uint32_t)c == tid)
            v = T(1);  // unit row standing in for a missing top row
        row[c] = v;
    }
    if (!is_top && valid)
#pragma unroll
        for (int c = 0; c < NB; ++c)
            if ((uint32_t)c < nb)
                backup[(size_t)(grow - k0) * NB + c] = row[c];
    bool bad = false;
#pragma unroll
    for (int j = 0; j < NB; ++j) {
        if (tid == (uint32_t)j) {
#pragma unroll
            for (int c = j; c < NB; ++c)
                U[j][c] = row[c];
            s_rcp[j] = T(1) / row[j];
            bad |= !(fabs(row[j]) > T(0));
        }
        __syncthreads();
        const bool act = is_top ? tid > (uint32_t)j : valid;
        if (act) {
            const T v = row[j];
            bad |= !(fabs(v) <= fabs(U[j][j]));
            const T x = v * s_rcp[j];
            row[j] = x;
#pragma unroll
            for (int c = j + 1; c < NB; ++c)
                row[c] -= x * U[j][c];
        }
    }
    if (__syncthreads_or(bad) && tid == 0)
        atomicExch(reject, 1);
    if (is_top) {
        if (blockIdx.x == 0 && valid)
#pragma unroll
            for (int c = 0; c < NB; ++c)
                if ((uint32_t)c < nb)
                    top_out[(size_t)tid * NB + c] = row[c];
    } else if (valid) {
#pragma unroll
        for (int c = 0; c < NB; ++c)
            if ((uint32_t)c < nb)
                A[(size_t)grow * lda + k0 + c] = row[c];
    }
}

// ---------------------------------------------------------------- 3. accept or pivot
// top_out: the speculative top block, committed here if the panel is accepted (FP32 path); NULL:
// the top block (and its identity pivots) is in A already, its old values in rows 0 .. 63 of backup.
// A rejected panel of at most stage_rows rows is factored in shared memory (stage_rows x (NB + 1)
// values of it): a column step is a chain of dependent passes over the panel, ~0.5 us each from
// shared memory and several from L2 (the last full panel of a closed body's bordered system, 65
// rows: 3.9 ms with one thread per row in global memory).
template <typename T>
__global__ void __launch_bounds__(1024) panel_pivot_kernel(uint32_t n, uint32_t k0, uint32_t nb, T* __restrict__ A,
                                                           uint32_t lda, const T* __restrict__ backup,
                                                           const T* __restrict__ top_out,
                                                           const int32_t* __restrict__ reject,
                                                           int32_t* __restrict__ ok, uint32_t panel,
                                                           int32_t* __restrict__ ipiv, int32_t* __restrict__ perm,
                                                           int32_t* __restrict__ info,
                                                           const T* __restrict__ backup_row, uint32_t stage_rows)
{
    extern __shared__ __align__(16) unsigned char pivot_smem[];
    __shared__ T s_val[32];
    __shared__ uint32_t s_idx[32];
    __shared__ uint32_t s_piv, s_pivs[NB], s_slot[NB];
    __shared__ int32_t s_top[NB], s_ext[NB];
    __shared__ T s_prow[NB];
    pvl::panel::grid_launch_next();  // trsm_kernel waits for this one's end
    const int bad = reject[panel];
    if (!bad) {
        if (threadIdx.x == 0)
            ok[panel] = 1;
        if (!top_out)
            return;
        for (uint32_t t = threadIdx.x; t < nb * nb; t += blockDim.x) {
            const uint32_t r = t / nb, c = t % nb;
            A[(size_t)(k0 + r) * lda + k0 + c] = top_out[(size_t)r * NB + c];
        }
        for (uint32_t j = threadIdx.x; j < nb; j += blockDim.x)
            ipiv[k0 + j] = (int32_t)(k0 + j);
        return;
    }
    if (threadIdx.x == 0)
        ok[panel] = 0;
    // restore what was overwritten (with top_out, the top block of A was not), in place or in shared
    // memory, then LAPACK getf2: first row of maximal |a|, swap, scale, update
    const uint32_t rows = n - k0;
    const bool staged = rows <= stage_rows;
    T* M = staged ? reinterpret_cast<T*>(pivot_smem) : A + (size_t)k0 * lda + k0;
    const size_t ldm = staged ? NB + 1 : lda;
    const uint32_t r_first = top_out ? nb : 0;
    for (size_t t = threadIdx.x; t < (size_t)rows * nb; t += blockDim.x) {
        const uint32_t r = (uint32_t)(t / nb), c = (uint32_t)(t % nb);
        if (r >= r_first)
            M[r * ldm + c] = backup[(size_t)r * NB + c];
        else if (staged)
            M[r * ldm + c] = A[(size_t)(k0 + r) * lda + k0 + c];
    }
    if (backup_row)  // the FP64 path also replaced the row block right of the panel by U12
        for (size_t t = threadIdx.x; t < (size_t)nb * (rows - nb); t += blockDim.x) {
            const uint32_t r = (uint32_t)(t / (rows - nb)), c = k0 + nb + (uint32_t)(t % (rows - nb));
            A[(size_t)(k0 + r) * lda + c] = backup_row[(size_t)r * n + c];
        }
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    for (uint32_t j = 0; j < nb; ++j) {
        T best = T(-1);
        uint32_t bidx = 0xFFFFFFFFu;
        for (uint32_t r = j + threadIdx.x; r < rows; r += blockDim.x) {
            const T v = fabs(M[r * ldm + j]);
            if (v > best) {
                best = v;
                bidx = r;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const T ov = __shfl_xor_sync(0xffffffffu, best, o);
            const uint32_t oi = __shfl_xor_sync(0xffffffffu, bidx, o);
            if (ov > best || (ov == best && oi < bidx)) {
                best = ov;
                bidx = oi;
            }
        }
        if (lane == 0) {
            s_val[warp] = best;
            s_idx[warp] = bidx;
        }
        __syncthreads();
        if (warp == 0) {
            T b = lane < n_warps ? s_val[lane] : T(-1);
            uint32_t bi = lane < n_warps ? s_idx[lane] : 0xFFFFFFFFu;
            for (int o = 16; o > 0; o >>= 1) {
                const T ov = __shfl_xor_sync(0xffffffffu, b, o);
                const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > b || (ov == b && oi < bi)) {
                    b = ov;
                    bi = oi;
                }
            }
            if (lane == 0) {
                bi = bi < rows ? bi : j;  // nothing compared greater (NaNs): no interchange
                s_piv = s_pivs[j] = bi;
                ipiv[k0 + j] = (int32_t)(k0 + bi);
            }
        }
        __syncthreads();
        const uint32_t p = s_piv;
        for (uint32_t c = threadIdx.x; c < nb; c += blockDim.x) {
            const T a = M[p * ldm + c];
            s_prow[c] = a;
            if (p != j) {
                M[p * ldm + c] = M[j * ldm + c];
                M[j * ldm + c] = a;
            }
        }
        __syncthreads();
        const T piv = s_prow[j];
        if (piv == T(0)) {
            if (threadIdx.x == 0)
                atomicCAS(info, 0, (int32_t)(k0 + j + 1));
            __syncthreads();
            continue;
        }
        const T rcp = T(1) / piv;
        for (uint32_t r = j + 1 + threadIdx.x; r < rows; r += blockDim.x)
            M[r * ldm + j] *= rcp;
        __syncthreads();
        // a warp per row, two columns per lane, kRowsAhead rows in flight
        constexpr uint32_t kRowsAhead = 4;
        const uint32_t c0 = j + 1 + lane, c1 = c0 + 32;
        const T p0 = c0 < nb ? s_prow[c0] : T(0), p1 = c1 < nb ? s_prow[c1] : T(0);
        for (uint32_t r = j + 1 + warp; r < rows; r += kRowsAhead * n_warps) {
            T l[kRowsAhead], a[kRowsAhead][2];
#pragma unroll
            for (uint32_t u = 0; u < kRowsAhead; ++u) {
                const uint32_t rr = r + u * n_warps;
                const bool in = rr < rows;
                l[u] = in ? M[rr * ldm + j] : T(0);
                a[u][0] = in && c0 < nb ? M[rr * ldm + c0] : T(0);
                a[u][1] = in && c1 < nb ? M[rr * ldm + c1] : T(0);
            }
#pragma unroll
            for (uint32_t u = 0; u < kRowsAhead; ++u) {
                const uint32_t rr = r + u * n_warps;
                if (rr < rows && c0 < nb)
                    M[rr * ldm + c0] = a[u][0] - l[u] * p0;
                if (rr < rows && c1 < nb)
                    M[rr * ldm + c1] = a[u][1] - l[u] * p1;
            }
        }
        __syncthreads();
    }
    if (staged)
        for (uint32_t t = threadIdx.x; t < rows * nb; t += blockDim.x) {
            const uint32_t r = t / nb, c = t % nb;
            A[(size_t)(k0 + r) * lda + k0 + c] = M[r * ldm + c];
        }
    // the panel's interchanges in perm: they touch its first nb entries (s_top) and those of the pivot
    // rows below (s_ext, one slot per distinct row: the first j that chose it)
    const uint32_t j = threadIdx.x;
    if (j < nb) {
        const uint32_t bi = s_pivs[j];
        uint32_t slot = j;
        for (uint32_t i = nb; i-- > 0;)
            if (s_pivs[i] == bi)
                slot = i;
        s_slot[j] = slot;
        s_top[j] = perm[k0 + j];
        s_ext[j] = perm[k0 + bi];
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (uint32_t i = 0; i < nb; ++i) {
            const uint32_t bi = s_pivs[i];
            int32_t& other = bi < nb ? s_top[bi] : s_ext[s_slot[i]];
            const int32_t t = s_top[i];
            s_top[i] = other;
            other = t;
        }
    __syncthreads();
    if (j < nb) {
        perm[k0 + j] = s_top[j];
        if (s_pivs[j] >= nb && s_slot[j] == j)
            perm[k0 + s_pivs[j]] = s_ext[j];
    }
}

// Rows that a rejected panel may have to be factored in shared memory.
constexpr uint32_t kPivotStageRows = 432;

template <typename T>
size_t pivot_smem(uint32_t rows)
{
    return rows <= kPivotStageRows ? (size_t)rows * (NB + 1) * sizeof(T) : 0;
}

// ---------------------------------------------------------------- 3. swaps + U12
// One thread per column outside the panel: apply the panel's interchanges (if any); columns
// right of the panel then solve L11 x = a (unit lower).  The 64 x 128 column block is staged
// through shared memory with coalesced row accesses; each thread keeps its column in
// registers during the substitution.
constexpr int kTrsmCols = 128;

template <typename T>
__global__ void __launch_bounds__(kTrsmCols, 1) trsm_kernel(uint32_t n, uint32_t k0, uint32_t nb, T* A,
                                                            uint32_t lda, const int32_t* ok, uint32_t panel,
                                                            const int32_t* ipiv, int fast_u12)
{
    if (fast_u12) {
        pvl::panel::grid_launch_next();  // the next panel's top_factor_kernel waits for this one's end
        pvl::panel::grid_wait();         // panel_pivot_kernel's
        if (*static_cast<const volatile int32_t*>(ok + panel))
            return;  // the FP64 path formed U12 = L11^-1 A12 already and nothing was interchanged
    }
    extern __shared__ double tsm_raw[];
    T* tsm = reinterpret_cast<T*>(tsm_raw);
    T(*L)[NB + 1] = reinterpret_cast<T(*)[NB + 1]>(tsm);                        // [NB][NB + 1]
    T(*X)[kTrsmCols + 1] = reinterpret_cast<T(*)[kTrsmCols + 1]>(tsm + NB * (NB + 1));  // [NB][129]
    const bool swapped = !ok[panel];
    const uint32_t t = blockIdx.x * kTrsmCols + threadIdx.x;
    const uint32_t n_out = n - nb;
    const uint32_t col = t < k0 ? t : t + nb;
    if (t < n_out && swapped)
        for (uint32_t j = 0; j < nb; ++j) {
            const uint32_t r1 = k0 + j, r2 = (uint32_t)ipiv[k0 + j];
            if (r1 != r2) {
                const T a = A[(size_t)r1 * lda + col];
                A[(size_t)r1 * lda + col] = A[(size_t)r2 * lda + col];
                A[(size_t)r2 * lda + col] = a;
            }
        }
    // the columns right of the panel start at k0 + nb; this CTA's first such column:
    const uint32_t c_first = blockIdx.x * kTrsmCols;  // in t-space
    if (c_first + kTrsmCols <= k0 || c_first >= n_out)
        return;  // CTA-uniform: only left-of-panel columns (already swapped) or none
    __syncthreads();  // swaps of this CTA's columns are visible before staging
    for (uint32_t e = threadIdx.x; e < NB * NB; e += kTrsmCols) {
        const uint32_t r = e / NB, c = e % NB;
        L[r][c] = (r < nb && c < nb) ? A[(size_t)(k0 + r) * lda + k0 + c] : T(0);
    }
    for (uint32_t e = threadIdx.x; e < NB * kTrsmCols; e += kTrsmCols) {
        const uint32_t r = e / kTrsmCols, c = e % kTrsmCols;
        const uint32_t tt = c_first + c;
        const uint32_t cc = tt < k0 ? tt : tt + nb;
        X[r][c] = (r < nb && tt < n_out && cc >= k0 + nb) ? A[(size_t)(k0 + r) * lda + cc] : T(0);
    }
    __syncthreads();
    T x[NB];
#pragma unroll
    for (int r = 0; r < NB; ++r)
        x[r] = X[r][threadIdx.x];
#pragma unroll
    for (int q = 0; q < NB - 1; ++q) {
        const T xq = x[q];
#pragma unroll
        for (int r = q + 1; r < NB; ++r)
            x[r] -= L[r][q] * xq;
    }
#pragma unroll
    for (int r = 0; r < NB; ++r)
        X[r][threadIdx.x] = x[r];
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < NB * kTrsmCols; e += kTrsmCols) {
        const uint32_t r = e / kTrsmCols, c = e % kTrsmCols;
        const uint32_t tt = c_first + c;
        const uint32_t cc = tt < k0 ? tt : tt + nb;
        if (r >= 1 && r < nb && tt < n_out && cc >= k0 + nb)
            A[(size_t)(k0 + r) * lda + cc] = X[r][c];
    }
}

// ---------------------------------------------------------------- FP64 panels and updates
// The FP64 factorisation first factors each panel without interchanges and then checks that
// partial pivoting would have made none: with no interchange before column j, GEPP keeps the
// diagonal in column j exactly when no entry below it is larger in magnitude at that moment,
// i.e. when every multiplier l_ij (i > j) has |l_ij| <= 1 (LAPACK's idamax returns the first
// maximal entry, and the diagonal comes first).  The multipliers and U12 are the blocked forms
// of getf2's and trsm's (lu_panel.cuh), equal to them up to rounding.

// One rectangle of the trailing update A22 -= L21 U12: C = rows row0 .. row0 + m, columns
// col0 .. col0 + nn; A = the panel's L21 (columns a_col ..) on C's rows, B = its U12 (rows
// b_row ..) on C's columns.  `ctas` CTAs, each group of a CTA a run of `per` 64 x 64 tiles.
struct UpdRect {
    uint32_t row0, col0, m, nn, a_col, b_row, per, ctas;
};

UpdRect upd_rect(uint32_t row0, uint32_t col0, uint32_t m, uint32_t nn, uint32_t k0, uint32_t max_ctas)
{
    const uint32_t tiles = blocks_for(m, pvl::dmma::kUpdTile) * blocks_for(nn, pvl::dmma::kUpdTile);
    UpdRect r{row0, col0, m, nn, k0, k0, 1, tiles};
    if (tiles > max_ctas) {  // fewer tiles than CTAs: one each, on SMs of their own
        r.per = blocks_for(tiles, pvl::dmma::kUpdGroups * max_ctas);
        r.ctas = blocks_for(blocks_for(tiles, r.per), pvl::dmma::kUpdGroups);
    }
    return r;
}

// One CTA per SM, each of its two groups a run of tiles in column-major order (dmma.cuh update_tiles).
template <bool VEC>
__global__ void __launch_bounds__(pvl::dmma::kUpdThreads, 1) dmma_update_kernel(double* __restrict__ A, uint32_t lda,
                                                                            UpdRect r)
{
    extern __shared__ __align__(16) double upd_smem[];
    auto* sm = reinterpret_cast<pvl::dmma::UpdSmem*>(upd_smem);
    constexpr uint32_t T = pvl::dmma::kUpdTile, G = pvl::dmma::kUpdGroupThreads;
    const uint32_t tiles = ((r.m + T - 1) / T) * ((r.nn + T - 1) / T);
    const uint32_t group = threadIdx.x / G, run = blockIdx.x + group * gridDim.x;
    const uint32_t t0 = min(tiles, run * r.per), t1 = min(tiles, t0 + r.per);
    pvl::dmma::update_tiles<VEC>(sm[group], (int)group, threadIdx.x % G, A, lda, r.row0, r.col0, r.m, r.nn, r.a_col,
                                 r.b_row, t0, t1);
}

// SMs that a trailing update (one CTA per SM) leaves to the next panel's kernels meanwhile: one for the
// diagonal block, and one for the first CTAs of the multipliers' kernel, which is started while that
// block is still being factored; the others follow as the update's CTAs end.  A share that grows as the block
// shrinks (8 and 256 columns' worth of the SMs, from before the chain's kernels were launched as
// dependents) no longer pays at any size: n = 2048 838 us with it, 827, 819, 821, 819 with 8, 4, 2 and
// 1 SMs; 3072 1646, 1619, 1608, 1599, 1598; 4096 2983, 2927, 2907, 2894, 2892; 8192 16956, 16615,
// 16536, 16506, 16500; up to 1536 all alike.
constexpr int kChainSms = 2;

// A kernel of the chain, allowed to start before the kernel ahead of it in the stream has ended
// (lu_panel.cuh grid_wait): its launch, and what it needs of older kernels only, run beside that
// one's end.  As ordinary launches n = 451 227 us, 1024 447, 2048 974, 4096 3036, 5121 5357; so 200,
// 387, 832, 2897, 5223.
cudaError_t launch_chained(const void* fn, dim3 grid, unsigned threads, void** args, size_t smem, cudaStream_t st)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, fn, args);
}

// A second stream and two events per thread and device for the look-ahead fork and join (a
// stream may take part in one capture at a time: per thread, since captures here are
// thread-local).  Created on first use in a context and kept; a new context (after a device
// reset) gets new ones.
struct SideStream {
    void* ctx = nullptr;
    cudaStream_t s = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
};

int side_stream(int dev, SideStream*& out)
{
    thread_local SideStream cache[64];
    if (dev < 0 || dev >= 64)
        return pvl_fail(PVL_ERR_ARG, "pvl_lu_factor: device %d out of range", dev);
    void* ctx = nullptr;
    if (int rc = pvl_current_context(&ctx))
        return rc;
    SideStream& c = cache[dev];
    if (!c.s || c.ctx != ctx) {
        c = SideStream{};
        PVL_CUDA_CHECK(cudaStreamCreateWithFlags(&c.s, cudaStreamNonBlocking));
        PVL_CUDA_CHECK(cudaEventCreateWithFlags(&c.fork, cudaEventDisableTiming));
        PVL_CUDA_CHECK(cudaEventCreateWithFlags(&c.join, cudaEventDisableTiming));
        c.ctx = ctx;
    }
    out = &c;
    return PVL_OK;
}

// ---------------------------------------------------------------- diagonal-block inverses
// With `reject` only the blocks of panels that took the pivoting fallback (the others' inverses
// came with their factors).  One CTA per kRB-row block b: threads 0..63 form column c of L_bb^-1 (unit lower, forward
// substitution), threads 64..127 column c of U_bb^-1 (backward substitution), each column
// held in registers.  A partial last block is padded with identity.  The wavefront solves
// then apply each diagonal block as one parallel matrix-vector product.
template <typename T>
__global__ void __launch_bounds__(2 * kRB, 1) diag_inverse_kernel(uint32_t n, const T* __restrict__ M,
                                                                  uint32_t lda, const int32_t* __restrict__ reject,
                                                                  T* __restrict__ inv)
{
    __shared__ T D[kRB][kRB + 1];
    const uint32_t b = blockIdx.x, r0 = b * kRB;
    if (reject && !reject[b])
        return;
    const uint32_t rows = min((uint32_t)kRB, n - r0);
    for (uint32_t e = threadIdx.x; e < kRB * kRB; e += blockDim.x) {
        const uint32_t r = e / kRB, c = e % kRB;
        D[r][c] = (r < rows && c < rows) ? M[(size_t)(r0 + r) * lda + r0 + c] : (r == c ? T(1) : T(0));
    }
    __syncthreads();
    const bool lower = threadIdx.x < kRB;
    const int c = (int)(threadIdx.x & (kRB - 1));
    T y[kRB];
    if (lower) {
#pragma unroll
        for (int r = 0; r < kRB; ++r)
            y[r] = r == c ? T(1) : T(0);
#pragma unroll
        for (int q = 0; q < kRB - 1; ++q) {
            const T yq = y[q];
#pragma unroll
            for (int r = q + 1; r < kRB; ++r)
                y[r] -= D[r][q] * yq;
        }
    } else {
#pragma unroll
        for (int r = 0; r < kRB; ++r)
            y[r] = r == c ? T(1) : T(0);
#pragma unroll
        for (int q = kRB - 1; q >= 0; --q) {
            const T yq = y[q] / D[q][q];
            y[q] = yq;
#pragma unroll
            for (int r = 0; r < q; ++r)
                y[r] -= D[r][q] * yq;
        }
    }
    T* out = inv + ((size_t)b * 2 + (lower ? 0 : 1)) * kRB * kRB;
#pragma unroll
    for (int r = 0; r < kRB; ++r)
        out[(size_t)r * kRB + c] = y[r];
}

// ---------------------------------------------------------------- solve
__global__ void gather_kernel(uint32_t n, const int32_t* __restrict__ perm, const double* __restrict__ b,
                              double* __restrict__ out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        out[i] = b[perm[i]];
}

// Blocked substitution with one launch per step and no inter-CTA waits (so that it can sit in a
// conditional body of a CUDA graph, where the wavefront's co-resident launch is not available):
// x_b = inv(D_bb) x_b for one diagonal block (one CTA), then the block's column slice updates
// the rows still to be solved (one warp per row).  Same inverted diagonal blocks as the wavefront.
template <bool LOWER>
__global__ void __launch_bounds__(kRB) diag_apply_kernel(uint32_t n, uint32_t b, const double* __restrict__ inv,
                                                         double* __restrict__ x)
{
    __shared__ double s[kRB];
    const uint32_t r0 = b * kRB, rows = min((uint32_t)kRB, n - r0), t = threadIdx.x;
    s[t] = t < rows ? x[r0 + t] : 0.0;
    __syncthreads();
    if (t < rows) {
        const double* D = inv + ((size_t)b * 2 + (LOWER ? 0 : 1)) * kRB * kRB + (size_t)t * kRB;
        double acc = 0.0;
#pragma unroll 8
        for (int c = 0; c < kRB; ++c)
            acc = fma(D[c], s[c], acc);
        x[r0 + t] = acc;
    }
}

template <bool LOWER>
__global__ void __launch_bounds__(256) block_update_kernel(uint32_t n, uint32_t b, const double* __restrict__ M,
                                                           uint32_t lda, double* __restrict__ x)
{
    const uint32_t c0 = b * kRB, cols = min((uint32_t)kRB, n - c0);
    const uint32_t first = LOWER ? c0 + cols : 0, count = LOWER ? n - first : c0;
    const uint32_t i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= count)
        return;
    const uint32_t r = first + i;
    const double* row = M + (size_t)r * lda + c0;
    double s = 0.0;
    for (uint32_t c = lane; c < cols; c += 32)
        s = fma(row[c], x[c0 + c], s);
    for (int o = 16; o > 0; o >>= 1)
        s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0)
        x[r] -= s;
}

int coresident_blocks(const void* fn, int threads, size_t smem)
{
    int dev = 0, sms = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess)
        return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, smem) != cudaSuccess)
        return 0;
    return sms * per;
}

}  // namespace

extern "C" size_t pvl_lu_workspace(uint32_t n) { return lu_ws_bytes(n); }

extern "C" int pvl_lu_factor(uint32_t n, double* A, uint32_t lda, int32_t* ipiv, int32_t* info, void* ws,
                             size_t ws_bytes, void* stream)
{
    if (n == 0)
        return PVL_OK;
    if (!A || !ipiv || !info || !ws)
        return pvl_fail(PVL_ERR_ARG, "pvl_lu_factor: null pointer argument");
    if (lda < n)
        return pvl_fail(PVL_ERR_ARG, "pvl_lu_factor: lda %u < n %u", lda, n);
    if (ws_bytes < lu_ws_bytes(n))
        return pvl_fail(PVL_ERR_ALLOC, "pvl_lu_factor: workspace %zu < %zu", ws_bytes, lu_ws_bytes(n));
    cudaStream_t st = (cudaStream_t)stream;
    LuWs w = carve(ws, n);
    const size_t trsm_smem = (size_t)(NB * (NB + 1) + NB * (kTrsmCols + 1)) * sizeof(double);
    const size_t upd_smem = pvl::dmma::kUpdGroups * sizeof(pvl::dmma::UpdSmem);
    int dev = 0, sms = 0;
    PVL_CUDA_CHECK(cudaGetDevice(&dev));
    PVL_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    SideStream* side = nullptr;
    if (int rc = side_stream(dev, side))
        return rc;
    // 16-byte operand copies need even row strides: a matrix of odd order is factored in a copy with
    // one and 128-byte aligned rows (5121: 7.0 ms in place with 8-byte copies, 5.2 so; 451: 213 and
    // 200 us); an odd last column is then copied with the padding after it.  An even order with an odd
    // stride keeps the 8-byte copies.
    const dim3 copy_grid(blocks_for(n, 256), std::min<uint32_t>(n, 1024));
    double* const given = A;
    const uint32_t given_lda = lda;
    if (even_stride(n)) {
        copy_matrix_kernel<<<copy_grid, 256, 0, st>>>(n, given, given_lda, w.even, even_stride(n));
        PVL_LAUNCH_CHECK();
        A = w.even;
        lda = even_stride(n);
    }
    const bool vec = lda % 2 == 0 && ((uintptr_t)A & 15u) == 0;
    const void* top_fn = vec ? (const void*)pvl::panel::top_factor_kernel<true>
                             : (const void*)pvl::panel::top_factor_kernel<false>;
    const void* apply_fn = vec ? (const void*)pvl::panel::panel_apply_kernel<true>
                               : (const void*)pvl::panel::panel_apply_kernel<false>;
    const void* upd_fn = vec ? (const void*)dmma_update_kernel<true> : (const void*)dmma_update_kernel<false>;
    const size_t top_smem = sizeof(pvl::panel::TopSmem);
    PVL_SMEM_OPTIN(trsm_kernel<double>, trsm_smem);
    PVL_SMEM_OPTIN(panel_pivot_kernel<double>, pivot_smem<double>(kPivotStageRows));
    PVL_SMEM_OPTIN(top_fn, top_smem);
    PVL_SMEM_OPTIN(apply_fn, pvl::panel::kApplySmem);
    PVL_SMEM_OPTIN(upd_fn, upd_smem);
    int32_t* perm = ipiv + n;
    PVL_CUDA_CHECK(cudaMemsetAsync(info, 0, sizeof(int32_t), st));
    init_perm_kernel<<<blocks_for(n, 256), 256, 0, st>>>(n, perm);
    PVL_LAUNCH_CHECK();
    const uint32_t n_panels = (n + NB - 1) / NB;
    // reject, and ok behind it: no panel counts as accepted before its own check
    PVL_CUDA_CHECK(cudaMemsetAsync(w.reject, 0, (size_t)((char*)w.tmp - (char*)w.reject), st));
    // Look-ahead: panel p's trailing update beyond panel p + 1 runs on the side stream, on all but
    // a share of the SMs, while panel p + 1's diagonal block, multipliers and row block (which
    // apply panel p's update to their own entries) run on `st`.  Panel p + 1's pivoting fallback,
    // whose interchanges reach every column, and everything after it wait for that update.
    bool pending = false;
    for (uint32_t p = 0; p < n_panels; ++p) {
        const uint32_t k0 = p * NB;
        const uint32_t nb = std::min<uint32_t>(NB, n - k0);
        const uint32_t below = n - k0 - nb;  // nonzero only for full panels (nb == NB)
        const int upd = p > 0;
        double* inv = w.inv + (size_t)p * 2 * NB * NB;
        int32_t* rj = w.reject + p;
        void* targs[] = {(void*)&n, (void*)&k0, (void*)&nb, (void*)&upd, (void*)&A, (void*)&lda, (void*)&w.backup,
                         (void*)&inv, (void*)&ipiv, (void*)&rj};
        if (p == 0)
            PVL_CUDA_CHECK(cudaLaunchKernel(top_fn, dim3(1), dim3(pvl::panel::kTopThreads), targs, top_smem, st));
        else  // after the previous panel's trsm_kernel
            PVL_CUDA_CHECK(launch_chained(top_fn, dim3(1), pvl::panel::kTopThreads, targs, top_smem, st));
        pvl_count_launch();
        if (below > 0) {
            const uint32_t tiles = blocks_for(below, pvl::panel::kApplyRows);
            void* args[] = {(void*)&n, (void*)&k0, (void*)&upd, (void*)&A, (void*)&lda, (void*)&inv, (void*)&w.backup,
                            (void*)&w.backup_row, (void*)&rj, (void*)&tiles};
            PVL_CUDA_CHECK(launch_chained(apply_fn, dim3(2 * tiles), pvl::panel::kApplyThreads, args,
                                          pvl::panel::kApplySmem, st));
            pvl_count_launch();
        }
        if (pending) {  // the previous panel's update
            PVL_CUDA_CHECK(cudaEventRecord(side->join, side->s));
            PVL_CUDA_CHECK(cudaStreamWaitEvent(st, side->join, 0));
            pending = false;
        }
        // an ordinary launch: it also waits for the side stream
        panel_pivot_kernel<double><<<1, 1024, pivot_smem<double>(n - k0), st>>>(
            n, k0, nb, A, lda, w.backup, nullptr, w.reject, w.ok, p, ipiv, perm, info,
            below > 0 ? w.backup_row : nullptr, kPivotStageRows);
        PVL_LAUNCH_CHECK();
        if (n > nb) {
            int fast = 1;
            void* sargs[] = {(void*)&n, (void*)&k0, (void*)&nb, (void*)&A, (void*)&lda, (void*)&w.ok, (void*)&p,
                             (void*)&ipiv, (void*)&fast};
            PVL_CUDA_CHECK(launch_chained((const void*)trsm_kernel<double>, dim3(blocks_for(n - nb, kTrsmCols)),
                                          kTrsmCols, sargs, trsm_smem, st));
            pvl_count_launch();
        }
        if (below <= NB)
            continue;  // the next panel is the last: it applies this update itself
        const uint32_t rest = k0 + 2 * NB;
        const UpdRect r = upd_rect(rest, rest, n - rest, n - rest, k0, (uint32_t)std::max(1, sms - kChainSms));
        PVL_CUDA_CHECK(cudaEventRecord(side->fork, st));
        PVL_CUDA_CHECK(cudaStreamWaitEvent(side->s, side->fork, 0));
        void* uargs[] = {(void*)&A, (void*)&lda, (void*)&r};
        PVL_CUDA_CHECK(cudaLaunchKernel(upd_fn, dim3(r.ctas), dim3(pvl::dmma::kUpdThreads), uargs, upd_smem, side->s));
        pvl_count_launch();
        pending = true;
    }
    if (pending) {
        PVL_CUDA_CHECK(cudaEventRecord(side->join, side->s));
        PVL_CUDA_CHECK(cudaStreamWaitEvent(st, side->join, 0));
    }
    diag_inverse_kernel<double><<<(n + kRB - 1) / kRB, 2 * kRB, 0, st>>>(n, A, lda, w.reject, w.inv);
    PVL_LAUNCH_CHECK();
    if (even_stride(n)) {
        copy_matrix_kernel<<<copy_grid, 256, 0, st>>>(n, A, lda, given, given_lda);
        PVL_LAUNCH_CHECK();
    }
    return PVL_OK;
}

extern "C" size_t pvl_lu_solve_workspace(uint32_t n) { return lu_ws_bytes(n); }

extern "C" int pvl_lu_solve(uint32_t n, const double* LU, uint32_t lda, const int32_t* ipiv, double* b,
                            int32_t* err, void* ws, size_t ws_bytes, void* stream)
{
    if (n == 0)
        return PVL_OK;
    if (!LU || !ipiv || !b || !ws || !err)
        return pvl_fail(PVL_ERR_ARG, "pvl_lu_solve: null pointer argument");
    if (ws_bytes < lu_ws_bytes(n))
        return pvl_fail(PVL_ERR_ALLOC, "pvl_lu_solve: workspace too small");
    const uint32_t nblk = (n + kRB - 1) / kRB;
    const void* fwd = (const void*)pvl::trsv::wavefront_kernel<true>;
    const void* bwd = (const void*)pvl::trsv::wavefront_kernel<false>;
    const size_t smem = pvl::trsv::kSmem;
    PVL_SMEM_OPTIN(fwd, smem);
    PVL_SMEM_OPTIN(bwd, smem);
    if ((int)nblk > coresident_blocks(fwd, kSolveThreads, smem) || (int)nblk > coresident_blocks(bwd, kSolveThreads, smem))
        return pvl_fail(PVL_ERR_ARG, "pvl_lu_solve: n = %u needs %u co-resident blocks", n, nblk);
    cudaStream_t st = (cudaStream_t)stream;
    LuWs w = carve(ws, n);
    // y = L^-1 P b, then x = U^-1 y (also into b); both start as "not ready" (trsv.cuh)
    double* y = w.backup;  // n x 64 doubles, free during the solve
    double* x = y + n;
    PVL_CUDA_CHECK(cudaMemsetAsync(err, 0, sizeof(int32_t), st));
    PVL_CUDA_CHECK(cudaMemsetAsync(y, pvl::trsv::kNotReadyByte, 2 * sizeof(double) * (size_t)n, st));
    const double* iv = w.inv;
    const int32_t* perm = ipiv + n;
    const int32_t* no_perm = nullptr;
    double* no_out = nullptr;
    int32_t* no_flags = nullptr;
    long long spin = pvl::trsv::kSpinLimit;
    int32_t skip = -1;
    void* fargs[] = {(void*)&n, (void*)&LU, (void*)&lda, (void*)&iv, (void*)&b, (void*)&perm, (void*)&y,
                     (void*)&no_out, (void*)&no_flags, (void*)&err, (void*)&spin, (void*)&skip};
    PVL_CUDA_CHECK(cudaLaunchCooperativeKernel(fwd, dim3(nblk), dim3(kSolveThreads), fargs, smem, st));
    pvl_count_launch();
    void* bargs[] = {(void*)&n, (void*)&LU, (void*)&lda, (void*)&iv, (void*)&y, (void*)&no_perm, (void*)&x,
                     (void*)&b, (void*)&no_flags, (void*)&err, (void*)&spin, (void*)&skip};
    PVL_CUDA_CHECK(cudaLaunchCooperativeKernel(bwd, dim3(nblk), dim3(kSolveThreads), bargs, smem, st));
    pvl_count_launch();
    return PVL_OK;
}

extern "C" int pvl_lu_solve_blocked(uint32_t n, const double* LU, uint32_t lda, const int32_t* ipiv, double* b,
                                    void* ws, size_t ws_bytes, void* stream)
{
    if (n == 0)
        return PVL_OK;
    if (!LU || !ipiv || !b || !ws)
        return pvl_fail(PVL_ERR_ARG, "pvl_lu_solve_blocked: null pointer argument");
    if (ws_bytes < lu_ws_bytes(n))
        return pvl_fail(PVL_ERR_ALLOC, "pvl_lu_solve_blocked: workspace too small");
    cudaStream_t st = (cudaStream_t)stream;
    LuWs w = carve(ws, n);
    const uint32_t nblk = (n + kRB - 1) / kRB;
    gather_kernel<<<blocks_for(n, 256), 256, 0, st>>>(n, ipiv + n, b, w.tmp);
    PVL_LAUNCH_CHECK();
    for (uint32_t k = 0; k < nblk; ++k) {
        diag_apply_kernel<true><<<1, kRB, 0, st>>>(n, k, w.inv, w.tmp);
        PVL_LAUNCH_CHECK();
        const uint32_t below = n - std::min(n, (k + 1) * kRB);
        if (below) {
            block_update_kernel<true><<<blocks_for(below, 8), 256, 0, st>>>(n, k, LU, lda, w.tmp);
            PVL_LAUNCH_CHECK();
        }
    }
    for (uint32_t k = nblk; k-- > 0;) {
        diag_apply_kernel<false><<<1, kRB, 0, st>>>(n, k, w.inv, w.tmp);
        PVL_LAUNCH_CHECK();
        if (k) {
            block_update_kernel<false><<<blocks_for(k * kRB, 8), 256, 0, st>>>(n, k, LU, lda, w.tmp);
            PVL_LAUNCH_CHECK();
        }
    }
    PVL_CUDA_CHECK(cudaMemcpyAsync(b, w.tmp, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
    return PVL_OK;
}

// ================================================================ FP32 LU (TF32 trailing update)
// The low-precision factorisation behind the mixed path's preconditioner.  Speculative panel
// (panel_spec_kernel), pivot and TRSM kernels instantiated for float, with the trailing update
// A22 -= L21 U12 on the tensor cores (U12 transposed into a K-major operand, then
// pvl_gemm_tf32: TMA-fed tcgen05 MMAs, TF32 products, FP32 accumulation).  The explicit inverse U^-1 L^-1 is then formed from the factors by blocked
// triangular inversion: the 64 x 64 diagonal-block products on CUDA cores in FP32, every
// rank-64 update on the tensor cores.  Applying the preconditioner is then one FP32
// matrix-vector product per Krylov iteration instead of two latency-bound triangular solves.
namespace {

// out[r][j] = sum_k D[r][k] in[k][j] for the 64 rows of a block (FP32, CUDA cores: the
// diagonal blocks of the inverse carry the O(1) entries whose TF32 rounding would dominate
// the preconditioner's error).  One thread per column, D staged in shared memory.
__global__ void __launch_bounds__(128) block_apply_kernel(uint32_t cols, const float* __restrict__ D,
                                                          const float* __restrict__ in, uint32_t ldi,
                                                          float* __restrict__ out, uint32_t ldo)
{
    __shared__ float sD[kRB][kRB];
    for (uint32_t e = threadIdx.x; e < kRB * kRB; e += blockDim.x)
        sD[e / kRB][e % kRB] = D[e];
    __syncthreads();
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cols)
        return;
    float x[kRB];
#pragma unroll
    for (int k = 0; k < kRB; ++k)
        x[k] = in[(size_t)k * ldi + j];
#pragma unroll 4
    for (int r = 0; r < kRB; ++r) {
        float s = 0.0f;
#pragma unroll
        for (int k = 0; k < kRB; ++k)
            s = fmaf(sD[r][k], x[k], s);
        out[(size_t)r * ldo + j] = s;
    }
}

__global__ void set_identity_kernel(uint32_t n, float* __restrict__ X, uint32_t ldx)
{
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (size_t)n * n)
        return;
    const uint32_t r = (uint32_t)(t / n), c = (uint32_t)(t % n);
    X[(size_t)r * ldx + c] = r == c ? 1.0f : 0.0f;
}

// out[r][perm[c]] = X[r][c]: the inverse's columns permuted, so that A^-1 b = out b.
__global__ void permute_columns_kernel(uint32_t n, const float* __restrict__ X, uint32_t ldx,
                                       const int32_t* __restrict__ perm, float* __restrict__ out, uint32_t ldo)
{
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (size_t)n * n)
        return;
    const uint32_t r = (uint32_t)(t / n), c = (uint32_t)(t % n);
    const uint32_t q = (uint32_t)perm[c];
    if (q < n)  // a valid factorisation never maps outside [0, n)
        out[(size_t)r * ldo + q] = X[(size_t)r * ldx + c];
}

// dst (cols x 64, row-major) = the transpose of the 64 x cols block src (leading dimension
// lds): the K-major form of a rank-64 update's right operand for the tensor-core GEMM.
__global__ void __launch_bounds__(256) transpose64_kernel(uint32_t cols, const float* __restrict__ src, uint32_t lds,
                                                          float* __restrict__ dst)
{
    __shared__ float t[32][33];
    const uint32_t c0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
    const uint32_t tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    for (uint32_t k = ty; k < 32; k += 8)
        t[k][tx] = c0 + tx < cols ? src[(size_t)(k0 + k) * lds + c0 + tx] : 0.0f;
    __syncthreads();
    for (uint32_t c = ty; c < 32; c += 8)
        if (c0 + c < cols)
            dst[(size_t)(c0 + c) * kRB + k0 + tx] = t[tx][c];
}

}  // namespace

extern "C" int pvl_gemm_tf32(uint32_t M, uint32_t N, uint32_t K, float alpha, const float* A, uint32_t lda,
                             const float* Bt, uint32_t ldbt, float beta, float* C, uint32_t ldc, int32_t* err,
                             void* stream);

namespace {
// C (M x cols) -= A (M x 64, lda) * B where B is the 64 x cols block at src (lds): B is
// transposed into bt (cols x 64) first, then the tensor-core GEMM runs on K-major operands.
int rank64_update(uint32_t M, uint32_t cols, const float* A, uint32_t lda, const float* src, uint32_t lds, float* bt,
                  float* C, uint32_t ldc, int32_t* err, cudaStream_t st)
{
    transpose64_kernel<<<dim3(blocks_for(cols, 32), kRB / 32), 256, 0, st>>>(cols, src, lds, bt);
    PVL_LAUNCH_CHECK();
    return pvl_gemm_tf32(M, cols, kRB, -1.0f, A, lda, bt, kRB, 1.0f, C, ldc, err, st);
}
}  // namespace

extern "C" size_t pvl_lu32_workspace(uint32_t n) { return lu_ws_bytes(n, true); }

extern "C" int pvl_lu32_factor(uint32_t n, float* A, uint32_t lda, int32_t* ipiv, int32_t* info, int32_t* err,
                               void* ws, size_t ws_bytes, void* stream)
{
    if (n == 0)
        return PVL_OK;
    if (!A || !ipiv || !info || !err || !ws)
        return pvl_fail(PVL_ERR_ARG, "pvl_lu32_factor: null pointer argument");
    if (lda < n || lda % 4 || ((uintptr_t)A & 15u))
        return pvl_fail(PVL_ERR_ARG, "pvl_lu32_factor: lda must be >= n and a multiple of 4, A 16-byte aligned");
    if (ws_bytes < lu_ws_bytes(n, true))
        return pvl_fail(PVL_ERR_ALLOC, "pvl_lu32_factor: workspace %zu < %zu", ws_bytes, lu_ws_bytes(n, true));
    cudaStream_t st = (cudaStream_t)stream;
    LuWs w = carve(ws, n);
    float* backup = reinterpret_cast<float*>(w.backup);
    float* top_out = reinterpret_cast<float*>(w.top_out);
    float* inv = reinterpret_cast<float*>(w.inv);
    float* ut = reinterpret_cast<float*>(w.backup_row);  // U12 transposed for the tensor-core updates
    const size_t trsm_smem = (size_t)(NB * (NB + 1) + NB * (kTrsmCols + 1)) * sizeof(float);
    PVL_SMEM_OPTIN(trsm_kernel<float>, trsm_smem);
    PVL_SMEM_OPTIN(panel_pivot_kernel<float>, pivot_smem<float>(kPivotStageRows));
    int32_t* perm = ipiv + n;
    PVL_CUDA_CHECK(cudaMemsetAsync(info, 0, sizeof(int32_t), st));
    PVL_CUDA_CHECK(cudaMemsetAsync(err, 0, sizeof(int32_t), st));
    init_perm_kernel<<<blocks_for(n, 256), 256, 0, st>>>(n, perm);
    PVL_LAUNCH_CHECK();
    const uint32_t n_panels = (n + NB - 1) / NB;
    PVL_CUDA_CHECK(cudaMemsetAsync(w.reject, 0, sizeof(int32_t) * (n_panels + 1), st));
    for (uint32_t p = 0; p < n_panels; ++p) {
        const uint32_t k0 = p * NB;
        const uint32_t nb = std::min<uint32_t>(NB, n - k0);
        const uint32_t below = n - k0 - nb;
        const uint32_t ctas = std::max<uint32_t>(1, (below + kSlabRows - 1) / kSlabRows);
        panel_spec_kernel<float><<<ctas, 2 * kSlabRows, 0, st>>>(n, k0, nb, A, lda, backup, top_out, w.reject + p);
        PVL_LAUNCH_CHECK();
        panel_pivot_kernel<float><<<1, 1024, pivot_smem<float>(n - k0), st>>>(
            n, k0, nb, A, lda, backup, top_out, w.reject, w.ok, p, ipiv, perm, info, nullptr, kPivotStageRows);
        PVL_LAUNCH_CHECK();
        if (n > nb) {
            trsm_kernel<float><<<blocks_for(n - nb, kTrsmCols), kTrsmCols, trsm_smem, st>>>(n, k0, nb, A, lda, w.ok, p,
                                                                                          ipiv, 0);
            PVL_LAUNCH_CHECK();
        }
        if (below > 0) {
            // every panel with rows below it is a full NB = 64 wide, so K = 64 (a multiple of 32)
            float* a22 = A + (size_t)(k0 + nb) * lda + k0 + nb;
            if (int r = rank64_update(below, below, A + (size_t)(k0 + nb) * lda + k0, lda, A + (size_t)k0 * lda + k0 + nb,
                                      lda, ut, a22, lda, err, st))
                return r;
        }
    }
    diag_inverse_kernel<float><<<(n + kRB - 1) / kRB, 2 * kRB, 0, st>>>(n, A, lda, nullptr, inv);
    PVL_LAUNCH_CHECK();
    return PVL_OK;
}

extern "C" int pvl_lu32_inverse(uint32_t n, const float* LU, uint32_t lda, const int32_t* perm, float* X,
                                uint32_t ldx, float* Y, uint32_t ldy, int32_t* err, void* ws, size_t ws_bytes,
                                void* stream)
{
    if (n == 0)
        return PVL_OK;
    if (!LU || !X || !Y || !err || !ws)
        return pvl_fail(PVL_ERR_ARG, "pvl_lu32_inverse: null pointer argument");
    if (n % kRB)
        return pvl_fail(PVL_ERR_ARG, "pvl_lu32_inverse: n = %u must be a multiple of %d", n, kRB);
    if (lda < n || ldx < n || ldy < n || lda % 4 || ldx % 4 || ldy % 4 ||
        (((uintptr_t)LU | (uintptr_t)X | (uintptr_t)Y) & 15u))
        return pvl_fail(PVL_ERR_ARG, "pvl_lu32_inverse: leading dimensions must be >= n and multiples of 4, "
                                     "arrays 16-byte aligned");
    if (ws_bytes < lu_ws_bytes(n, true))
        return pvl_fail(PVL_ERR_ALLOC, "pvl_lu32_inverse: workspace too small");
    cudaStream_t st = (cudaStream_t)stream;
    LuWs w = carve(ws, n);
    const float* inv = reinterpret_cast<const float*>(w.inv);  // written by pvl_lu32_factor
    float* bt = reinterpret_cast<float*>(w.backup_row);         // transposed update operands
    const uint32_t nblk = n / kRB;
    // forward: Y = L^-1, with X as the working right-hand side (starts as I)
    set_identity_kernel<<<blocks_for((size_t)n * n, 256), 256, 0, st>>>(n, X, ldx);
    PVL_LAUNCH_CHECK();
    PVL_CUDA_CHECK(cudaMemset2DAsync(Y, (size_t)ldy * sizeof(float), 0, (size_t)n * sizeof(float), n, st));
    for (uint32_t k = 0; k < nblk; ++k) {
        const uint32_t r0 = k * kRB, cols = r0 + kRB;  // L^-1 is zero right of the diagonal block
        block_apply_kernel<<<blocks_for(cols, 128), 128, 0, st>>>(cols, inv + (size_t)k * 2 * kRB * kRB,
                                                                 X + (size_t)r0 * ldx, ldx, Y + (size_t)r0 * ldy, ldy);
        PVL_LAUNCH_CHECK();
        if (cols < n)
            if (int r = rank64_update(n - cols, cols, LU + (size_t)cols * lda + r0, lda, Y + (size_t)r0 * ldy, ldy, bt,
                                      X + (size_t)cols * ldx, ldx, err, st))
                return r;
    }
    // backward: X = U^-1 Y, with Y as the working right-hand side
    for (uint32_t kk = nblk; kk-- > 0;) {
        const uint32_t r0 = kk * kRB;
        block_apply_kernel<<<blocks_for(n, 128), 128, 0, st>>>(n, inv + ((size_t)kk * 2 + 1) * kRB * kRB,
                                                              Y + (size_t)r0 * ldy, ldy, X + (size_t)r0 * ldx, ldx);
        PVL_LAUNCH_CHECK();
        if (r0 > 0)
            if (int r = rank64_update(r0, n, LU + r0, lda, X + (size_t)r0 * ldx, ldx, bt, Y, ldy, err, st))
                return r;
    }
    if (perm) {
        // A^-1 = U^-1 L^-1 P with (P b)[i] = b[perm[i]]: fold P into the columns
        permute_columns_kernel<<<blocks_for((size_t)n * n, 256), 256, 0, st>>>(n, X, ldx, perm, Y, ldy);
        PVL_LAUNCH_CHECK();
        PVL_CUDA_CHECK(cudaMemcpy2DAsync(X, (size_t)ldx * sizeof(float), Y, (size_t)ldy * sizeof(float),
                                         (size_t)n * sizeof(float), n, cudaMemcpyDeviceToDevice, st));
    }
    return PVL_OK;
}
