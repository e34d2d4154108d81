// The FP64 LU's panel kernels (lu.cu): the 64 x 64 diagonal block of a panel with its inverses,
// and the panel's multipliers and row block, each fused with the previous panel's update of the
// same entries (so that no separate launch updates the next panel before it is factored).
//
// Notation: panel p = columns k0 .. k0 + 63.  On entry every block of panel p's row and column
// holds the updates of panels 0 .. p - 2; both kernels apply panel p - 1's (L[:, p-1] U[p-1, :])
// themselves.  What they overwrite is backed up in updated form, so a panel in which partial
// pivoting would have interchanged rows can be restored and refactored (panel_pivot_kernel).
#pragma once

#include <cstdint>

#include "dmma.cuh"

namespace pvl {
namespace panel {

using dmma::kPad;

constexpr int NB = 64;                 // panel width
constexpr int kTopThreads = 256;
constexpr double kPivotLo = 0x1p-1000, kPivotHi = 0x1p+1000;

// 1/p for a pivot with kPivotLo <= |p| <= kPivotHi: the hardware's approximate reciprocal r
// (rcp.approx.ftz.f64, relative error d < 2^-19) refined by one third-order step of the
// geometric series 1/p = r / (1 - e), e = 1 - p r:  r + r (e + e^2) = (1/p)(1 - d^3), within an
// ulp of the rounded quotient.  Pivots outside the range take the exact (pivoting) path.
__device__ __forceinline__ double pivot_rcp(double p)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(p));
    const double e = fma(-p, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

__device__ __forceinline__ void mma8x8x4(double2& c, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c.x), "+d"(c.y)
                 : "d"(a), "d"(b));
}

// acc (MT x NT tiles of 16 x 8) += A (rows from as, stride kPad) * B (64 x ., from bs, stride kPad)
template <int MT, int NT>
__device__ __forceinline__ void mma_k64(double (&acc)[MT][NT][4], const double* as, const double* bs, uint32_t g,
                                        uint32_t t)
{
#pragma unroll
    for (int k0 = 0; k0 < NB; k0 += 8) {
        double af[MT][4], bf[NT][2];
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const double* p = as + (16 * i + g) * kPad + k0 + t;
            af[i][0] = p[0];
            af[i][1] = p[8 * kPad];
            af[i][2] = p[4];
            af[i][3] = p[8 * kPad + 4];
        }
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            const double* p = bs + (k0 + t) * kPad + 8 * j + g;
            bf[j][0] = p[0];
            bf[j][1] = p[4 * kPad];
        }
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
                dmma::mma16x8x8(acc[i][j], af[i], bf[j]);
    }
}

// acc = -C over the warp's 16 MT x 8 NT entries (rows from `row`, columns from `col`, valid below
// m_end / n_end); entries outside are 0.
template <int MT, int NT, bool VEC>
__device__ __forceinline__ void load_neg(double (&acc)[MT][NT][4], const double* C, uint32_t ldc, uint32_t row,
                                         uint32_t col, uint32_t m_end, uint32_t n_end, uint32_t g, uint32_t t)
{
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t r = row + 16 * i + g + 8 * h, c = col + 8 * j + 2 * t;
                double v0 = 0.0, v1 = 0.0;
                if (r < m_end) {
                    const double* p = C + (size_t)r * ldc + c;
                    if (VEC && c + 1 < n_end) {
                        const double2 v = *reinterpret_cast<const double2*>(p);
                        v0 = v.x;
                        v1 = v.y;
                    } else {
                        if (c < n_end)
                            v0 = p[0];
                        if (c + 1 < n_end)
                            v1 = p[1];
                    }
                }
                acc[i][j][2 * h] = -v0;
                acc[i][j][2 * h + 1] = -v1;
            }
}

// ---------------------------------------------------------------- the diagonal block
// One CTA of 8 warps: the updated 64 x 64 diagonal block factored without interchanges, with
// X = L^-1 and Y = U^-1 formed by the same eliminations, in eight steps of 8 columns.  Step k:
//   * warps 0-3: every thread loads the 8 x 8 diagonal block and factors it in registers,
//     redundantly (the chain of 8 pivots then needs no exchange between lanes).  Thread r < 64
//     solves row r of column block k against U_kk -- a row of T below the block (multipliers,
//     checked), a row of Y in or above it -- and thread 64 + c column c of row block k against
//     L_kk -- a column of T right of the block, of X in or left of it.
//   * the rank-8 update of everything else, 8 x 8 tiles on the FP64 tensor cores: T[i][j], X[i][j]
//     and Y[i][j] -= left(i) right(j) with left(i) = T or Y block (i, k), right(j) = T or X block
//     (k, j).  Warps 0-3 take the tiles of row block and column block k + 1 and go on to step
//     k + 1; warps 4-7 take the rest meanwhile (disjoint blocks).
// What bounds it is latency, not the operations: measured with clock stamps, ~3000 cycles until the
// operands are there, 4300 for the corner's product on one SM, eight steps of ~2000 (the 8 x 8
// block 950, the solves 200, the barrier 200, the next row and column blocks 600), 3500 for the
// stores; 19-21 us a block against 37 us (plus a separate update launch) with one barrier per column.
constexpr int kTopPad = 132;  // row stride of xt in doubles (132 = 4 mod 16, as kPad)
struct __align__(16) TopSmem {
    double xt[NB][kTopPad];  // X in columns 0 .. 63, T in columns 64 .. 127
    double y[NB][kPad];
};
constexpr int kYAt = NB * kTopPad;  // y's place in the same array of doubles

// N 8 x 8 tiles dst -= left right (K = 8), given the lane's positions in m of left (g, t), right (t, g)
// and dst (g, 2 t), g = lane / 4, t = lane % 4; tile u is stored where store(u).  All loads, then the
// two products of every tile in turn (one after the other they would wait for each other), then
// the stores.
template <int N, typename F>
__device__ __forceinline__ void tiles(double* m, const int (&dst)[N], const int (&left)[N], const int (&right)[N],
                                      F store)
{
    double2 c[N];
    double a[N][2], b[N][2];
#pragma unroll
    for (int u = 0; u < N; ++u) {
        c[u] = *reinterpret_cast<const double2*>(m + dst[u]);
        a[u][0] = -m[left[u]];
        a[u][1] = -m[left[u] + 4];
        b[u][0] = m[right[u]];
        b[u][1] = m[right[u] + 4 * kTopPad];
    }
#pragma unroll
    for (int u = 0; u < N; ++u)
        mma8x8x4(c[u], a[u][0], b[u][0]);
#pragma unroll
    for (int u = 0; u < N; ++u)
        mma8x8x4(c[u], a[u][1], b[u][1]);
#pragma unroll
    for (int u = 0; u < N; ++u)
        if (store(u))
            *reinterpret_cast<double2*>(m + dst[u]) = c[u];
}

// Programmatic dependent launch (the chain's kernels may be started before the one ahead of them in
// the stream has ended): wait until it has, its writes visible; and let the next kernel start.
// Every kernel launched so waits before it ends, so its own end implies all earlier ones'.
// No parameter of a kernel that waits so is __restrict__: the kernel ahead still writes through the
// same addresses when this one has started, and the qualifier would let the compiler read them
// through the non-coherent path or ahead of the wait.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ void panel_group_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// The high word of |v|: an order on magnitudes to 2^-20, compared on the integer pipe.
__device__ __forceinline__ int mag_hi(double v) { return __double2hiint(v) & 0x7FFFFFFF; }

// The step after which panel_apply_kernel may start: late, since its waiting CTAs hold SMs that the
// bulk update beside this kernel would take, but early enough for its loads and first product (after
// steps 3, 4 or 5: n = 1024 387 us, 4096 2898; after 6: 392, 2916; after 7, the last: 397, 2923).
constexpr int kTopTrigger = 5;

// update: panel p - 1 exists.  backup: rows 0 .. 63 of the panel's backup.  inv: (2, 64, 64), L^-1
// and U^-1 of this block (a partial block padded with identity).
template <bool VEC>
__global__ void __launch_bounds__(kTopThreads, 1) top_factor_kernel(uint32_t n, uint32_t k0, uint32_t nb, int update,
                                                                    double* A, uint32_t lda, double* backup,
                                                                    double* inv, int32_t* ipiv, int32_t* reject)
{
    extern __shared__ __align__(16) double top_smem[];
    TopSmem& s = *reinterpret_cast<TopSmem*>(top_smem);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t g = lane >> 2, t4 = lane & 3;
    const uint32_t wm0 = (warp >> 2) * 32, wn0 = (warp & 3) * 16;
    double acc[2][2][4];
    double* m = top_smem;                 // xt, then y
    double* ls = m;                       // L[p, p-1] and U[p-1, p] (stride kPad), before xt and y are needed
    double* us = ls + NB * kPad;
    static_assert(sizeof(TopSmem) >= 2 * NB * kPad * sizeof(double), "the corner's operands fit");
    grid_wait();
    if (update) {
        dmma::stage_tile<NB, NB, VEC, kTopThreads>(ls, A, lda, k0, k0 + nb, k0 - NB, k0, tid);
        dmma::stage_tile<NB, NB, VEC, kTopThreads>(us, A, lda, k0 - NB, k0, k0, k0 + nb, tid);
    }
    load_neg<2, 2, VEC>(acc, A + (size_t)k0 * lda + k0, lda, wm0, wn0, nb, nb, g, t4);
    dmma::cp_async_wait_all();
    __syncthreads();
    if (update) {
        mma_k64<2, 2>(acc, ls + wm0 * kPad, us + wn0, g, t4);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t r = wm0 + g + 16 * i + 8 * h, c = wn0 + 2 * t4 + 8 * j;
                const double2 v = make_double2(-acc[i][j][2 * h], -acc[i][j][2 * h + 1]);
                if (r < nb)  // the backup has n rows
                    *reinterpret_cast<double2*>(backup + r * NB + c) = v;  // columns past nb: never read
                *reinterpret_cast<double2*>(&s.xt[r][NB + c]) = v;
                const double2 e = make_double2(r == c ? 1.0 : 0.0, r == c + 1 ? 1.0 : 0.0);
                *reinterpret_cast<double2*>(&s.xt[r][c]) = e;
                *reinterpret_cast<double2*>(&s.y[r][c]) = e;
            }
    if (nb < NB) {  // a partial block (the last): padded with identity
        __syncthreads();
        for (uint32_t e = tid; e < NB * NB; e += kTopThreads) {
            const uint32_t r = e / NB, c = e % NB;
            if (r >= nb || c >= nb)
                s.xt[r][NB + c] = r == c ? 1.0 : 0.0;
        }
    }
    __syncthreads();
    int worst = 0;   // largest multiplier (mag_hi)
    int lo = 0x7FFFFFFF, hi = 0;  // smallest and largest pivot
#pragma unroll 1
    for (int k = 0; k < NB / 8; ++k) {
        const int b = 8 * k;
        if (warp < 4) {
            double D[8][8], rc[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    const double2 v = *reinterpret_cast<const double2*>(&s.xt[b + i][NB + b + j]);
                    D[i][j] = v.x;
                    D[i][j + 1] = v.y;
                }
            const bool is_row = tid < 64;
            const int q = (int)(tid & 63u);
            const bool beyond = q >= b + 8;  // row below / column right of the diagonal block
            double x[8];
            double* px = is_row ? (beyond ? &s.xt[q][NB + b] : &s.y[q][b]) : &s.xt[b][q + (beyond ? NB : 0)];
            if (is_row) {
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    const double2 v = *reinterpret_cast<const double2*>(px + i);
                    x[i] = v.x;
                    x[i + 1] = v.y;
                }
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    x[i] = px[i * kTopPad];
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                lo = min(lo, mag_hi(D[j][j]));
                hi = max(hi, mag_hi(D[j][j]));
                rc[j] = pivot_rcp(D[j][j]);
#pragma unroll
                for (int i = j + 1; i < 8; ++i) {
                    D[i][j] *= rc[j];
                    worst = max(worst, mag_hi(D[i][j]));
                }
#pragma unroll
                for (int i = j + 1; i < 8; ++i)
#pragma unroll
                    for (int c = j + 1; c < 8; ++c)
                        D[i][c] = fma(-D[i][j], D[j][c], D[i][c]);
            }
            if (is_row) {  // x U_kk = row
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    x[j] *= rc[j];
#pragma unroll
                    for (int c = j + 1; c < 8; ++c)
                        x[c] = fma(-x[j], D[j][c], x[c]);
                }
                if (beyond) {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        worst = max(worst, mag_hi(x[j]));
                }
#pragma unroll
                for (int i = 0; i < 8; i += 2)
                    *reinterpret_cast<double2*>(px + i) = make_double2(x[i], x[i + 1]);
            } else {  // L_kk x = column (unit lower)
#pragma unroll
                for (int j = 0; j < 7; ++j)
#pragma unroll
                    for (int i = j + 1; i < 8; ++i)
                        x[i] = fma(-D[i][j], x[j], x[i]);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    px[i * kTopPad] = x[i];
            }
            panel_group_sync();  // every thread of the group has read the diagonal block
            if (is_row) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (q == b + i) {
#pragma unroll
                        for (int j = 0; j < 8; j += 2)
                            *reinterpret_cast<double2*>(&s.xt[q][NB + b + j]) = make_double2(D[i][j], D[i][j + 1]);
                    }
            }
        }
        __syncthreads();  // step k's rows and columns are final, update k - 1 is complete
        if (k == kTopTrigger)
            grid_launch_next();  // panel_apply_kernel: its first product needs nothing of this block
        if (k == NB / 8 - 1)
            break;
        // Column j of the update: X's column block j for j <= k, T's for j > k; the rows below take all
        // eight, those above (Y) the T columns, each with row block k of the same column.
        const int right0 = (b + (int)t4) * kTopPad + (int)g;
        if (warp < 2) {  // row block k + 1, four columns each
            int d[4], l[4], r[4];
            const int row = (b + 8 + (int)g) * kTopPad;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = 4 * (int)warp + u, o = 8 * j + (j > k ? NB : 0);
                d[u] = row + o + 2 * (int)t4;
                l[u] = row + NB + b + (int)t4;
                r[u] = right0 + o;
            }
            tiles<4>(m, d, l, r, [](int) { return true; });
        } else if (warp < 4) {  // column block k + 1, four rows each
            int d[4], l[4], r[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = 4 * (int)(warp - 2) + u;
                const int row = i > k ? (8 * i + (int)g) * kTopPad + NB : kYAt + (8 * i + (int)g) * kPad;
                d[u] = row + b + 8 + 2 * (int)t4;
                l[u] = row + b + (int)t4;
                r[u] = right0 + b + 8 + NB;
            }
            tiles<4>(m, d, l, r, [&](int u) { return 4 * (int)(warp - 2) + u != k + 1; });
        } else {
            const int w = (int)warp - 4, mm = 6 - k;  // column blocks k + 2 .. 7
#pragma unroll 1
            for (int i = k + 2 + w; i < 8; i += 4) {
                const int row = (8 * i + (int)g) * kTopPad;
#pragma unroll 1
                for (int h = 0; h < 8; h += 4) {
                    int d[4], l[4], r[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int o = 8 * (h + u) + (h + u > k ? NB : 0);
                        d[u] = row + o + 2 * (int)t4;
                        l[u] = row + NB + b + (int)t4;
                        r[u] = right0 + o;
                    }
                    tiles<4>(m, d, l, r, [&](int u) { return h + u != k + 1; });
                }
            }
            const int n = (k + 1) * mm;
            if (w < n) {  // at most 12 tiles of Y: three per warp (an absent one repeats the first, unstored)
                int d[3], l[3], r[3];
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    const int e = w + 4 * u < n ? w + 4 * u : w, j = k + 2 + e % mm;
                    const int row = kYAt + (8 * (e / mm) + (int)g) * kPad;
                    d[u] = row + 8 * j + 2 * (int)t4;
                    l[u] = row + b + (int)t4;
                    r[u] = right0 + 8 * j + NB;
                }
                tiles<3>(m, d, l, r, [&](int u) { return w + 4 * u < n; });
            }
        }
        if (warp < 4)
            panel_group_sync();
    }
    // the range of a pivot that pivot_rcp takes, and the limit of a multiplier (both to the high word:
    // what lies within 2^-20 of a bound takes the pivoting path, which is always right)
    const bool bad = lo <= __double2hiint(kPivotLo) || hi >= __double2hiint(kPivotHi) ||
                     worst >= __double2hiint(dmma::kMultLimit);
    if (__syncthreads_or(warp < 4 && bad) && tid == 0)
        atomicExch(reject, 1);
    const uint32_t c = 2 * lane;
#pragma unroll
    for (int u = 0; u < 8; ++u) {  // row warp + 8 u, two columns per lane
        const uint32_t r = warp + 8 * u;
        const double2 x = *reinterpret_cast<const double2*>(&s.xt[r][c]);
        const double2 y = *reinterpret_cast<const double2*>(&s.y[r][c]);
        const double2 v = *reinterpret_cast<const double2*>(&s.xt[r][NB + c]);
        *reinterpret_cast<double2*>(inv + r * NB + c) = x;
        *reinterpret_cast<double2*>(inv + NB * NB + r * NB + c) = y;
        double* o = A + (size_t)(k0 + r) * lda + k0 + c;
        if (VEC && c + 1 < nb) {
            if (r < nb)
                *reinterpret_cast<double2*>(o) = v;
        } else if (r < nb) {
            if (c < nb)
                o[0] = v.x;
            if (c + 1 < nb)
                o[1] = v.y;
        }
    }
    if (tid < nb)
        ipiv[k0 + tid] = (int32_t)(k0 + tid);  // rewritten by the pivoting fallback
}

// ---------------------------------------------------------------- multipliers and row block
// CTAs 0 .. n_ltiles - 1: R rows of the panel's columns below the diagonal block,
//   A21 := (A21 - L[., p-1] U[p-1, p]) U11^-1   (the multipliers, each checked);
// the rest: R columns of the panel's row block,
//   A12 := L11^-1 (A12 - L[p, p-1] U[p-1, .]).
// 4 warps; the updated operand goes through shared memory between the two products, and to the
// backup.  The first product reads only what older panels left, so it runs before grid_wait, beside
// the end of top_factor_kernel.  R = 16 at every size: the shortest chain per CTA, and the few SMs that
// the bulk update leaves are shared most evenly (16, 32, 64 rows: n = 451 204, 214, 252 us; 2048 832, 897,
// 1072; 4096 2921, 3084, 3518; 8192 16572, 16703, 17688).
constexpr int kApplyRows = 16;
constexpr int kApplyThreads = 128;
constexpr size_t kApplySmem = (size_t)3 * NB * kPad * sizeof(double);

template <bool VEC>
__global__ void __launch_bounds__(kApplyThreads, 2) panel_apply_kernel(uint32_t n, uint32_t k0, int update,
                                                                       double* A, uint32_t lda, const double* inv,
                                                                       double* backup, double* backup_row, int32_t* reject,
                                                                       uint32_t n_ltiles)
{
    constexpr int R = kApplyRows;
    extern __shared__ __align__(16) double apply_smem[];
    double* s0 = apply_smem;              // L: R x 64 rows / U: 64 x 64 of L[p, p-1]
    double* s1 = s0 + NB * kPad;          // U[p-1, .] (64 x 64 / 64 x R)
    double* s2 = s1 + NB * kPad;          // U11^-1 / L11^-1
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t g = lane >> 2, t4 = lane & 3;
    const uint32_t base = k0 + NB;
    const bool lower = blockIdx.x < n_ltiles;
    const uint32_t e0 = base + (lower ? blockIdx.x : blockIdx.x - n_ltiles) * R;  // first row / column
    const uint32_t cnt = min((uint32_t)R, n - e0);
    bool bad = false;
    if (lower) {
        constexpr int NT = 2;  // every warp: 16 rows x 16 columns
        const uint32_t wn0 = warp * 16;
        double acc[1][NT][4];
        if (update) {
            dmma::stage_tile<R, NB, VEC, kApplyThreads>(s0, A, lda, e0, e0 + cnt, k0 - NB, k0, tid);
            dmma::stage_tile<NB, NB, VEC, kApplyThreads>(s1, A, lda, k0 - NB, k0, k0, base, tid);
        }
        load_neg<1, NT, VEC>(acc, A + (size_t)e0 * lda + k0, lda, 0, wn0, cnt, NB, g, t4);
        dmma::cp_async_wait_all();
        __syncthreads();
        if (update)
            mma_k64<1, NT>(acc, s0, s1 + wn0, g, t4);
        grid_wait();
        dmma::stage_tile<NB, NB, true, kApplyThreads>(s2, inv + NB * NB, NB, 0, NB, 0, NB, tid);
        __syncthreads();  // s0 is read no more
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t r = g + 8 * h, c = wn0 + 8 * j + 2 * t4;
                const double2 v = make_double2(-acc[0][j][2 * h], -acc[0][j][2 * h + 1]);
                *reinterpret_cast<double2*>(s0 + r * kPad + c) = v;
                if (r < cnt)
                    *reinterpret_cast<double2*>(backup + (size_t)(e0 + r - k0) * NB + c) = v;
                acc[0][j][2 * h] = acc[0][j][2 * h + 1] = 0.0;
            }
        dmma::cp_async_wait_all();
        __syncthreads();
        mma_k64<1, NT>(acc, s0, s2 + wn0, g, t4);
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t r = g + 8 * h, c = wn0 + 8 * j + 2 * t4;
                if (r >= cnt)
                    continue;
                const double v0 = acc[0][j][2 * h], v1 = acc[0][j][2 * h + 1];
                bad |= !(fabs(v0) < dmma::kMultLimit) || !(fabs(v1) < dmma::kMultLimit);
                double* o = A + (size_t)(e0 + r) * lda + k0 + c;
                if (VEC) {
                    *reinterpret_cast<double2*>(o) = make_double2(v0, v1);
                } else {
                    o[0] = v0;
                    o[1] = v1;
                }
            }
    } else {
        constexpr int NT = R / 8;  // every warp: 16 rows x R columns
        const uint32_t wm0 = warp * 16;
        double acc[1][NT][4];
        if (update) {
            dmma::stage_tile<NB, NB, VEC, kApplyThreads>(s0, A, lda, k0, base, k0 - NB, k0, tid);
            dmma::stage_tile<NB, R, VEC, kApplyThreads>(s1, A, lda, k0 - NB, k0, e0, e0 + cnt, tid);
        }
        load_neg<1, NT, VEC>(acc, A + (size_t)k0 * lda + e0, lda, wm0, 0, NB, cnt, g, t4);
        dmma::cp_async_wait_all();
        __syncthreads();
        if (update)
            mma_k64<1, NT>(acc, s0 + wm0 * kPad, s1, g, t4);
        grid_wait();
        dmma::stage_tile<NB, NB, true, kApplyThreads>(s2, inv, NB, 0, NB, 0, NB, tid);
        __syncthreads();  // s1 is read no more
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t r = wm0 + g + 8 * h, c = 8 * j + 2 * t4;
                const double v0 = -acc[0][j][2 * h], v1 = -acc[0][j][2 * h + 1];
                *reinterpret_cast<double2*>(s1 + r * kPad + c) = make_double2(v0, v1);
                double* bk = backup_row + (size_t)r * n + e0 + c;
                if (c < cnt)
                    bk[0] = v0;
                if (c + 1 < cnt)
                    bk[1] = v1;
                acc[0][j][2 * h] = acc[0][j][2 * h + 1] = 0.0;
            }
        dmma::cp_async_wait_all();
        __syncthreads();
        mma_k64<1, NT>(acc, s2 + wm0 * kPad, s1, g, t4);
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t r = wm0 + g + 8 * h, c = 8 * j + 2 * t4;
                double* o = A + (size_t)(k0 + r) * lda + e0 + c;
                const double v0 = acc[0][j][2 * h], v1 = acc[0][j][2 * h + 1];
                if (VEC && c + 1 < cnt) {
                    *reinterpret_cast<double2*>(o) = make_double2(v0, v1);
                } else {
                    if (c < cnt)
                        o[0] = v0;
                    if (c + 1 < cnt)
                        o[1] = v1;
                }
            }
    }
    if (lower && __syncthreads_or(bad) && tid == 0)
        atomicExch(reject, 1);
}

}  // namespace panel
}  // namespace pvl
