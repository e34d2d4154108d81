// FP64 tensor-core tiles (mma.sync m16n8k8 .f64) for the LU's rank-64 products.
//
// Operands are staged in shared memory by cp.async, row-major (8-byte copies when a leading
// dimension is odd, 16-byte ones otherwise), rows padded to 68 doubles, so the fragment loads
// of a half-warp (groupID 0..3, thread-in-group 0..3) hit 16 distinct 8-byte bank pairs.
// Fragment layout of mma.m16n8k8 .f64 (g = lane / 4, t = lane % 4):
//   A 16 x 8: a0 (g, t), a1 (g + 8, t), a2 (g, t + 4), a3 (g + 8, t + 4)
//   B 8 x 8:  b0 (t, g), b1 (t + 4, g)
//   C 16 x 8: c0 (g, 2t), c1 (g, 2t + 1), c2 (g + 8, 2t), c3 (g + 8, 2t + 1)
#pragma once

#include <cstdint>

namespace pvl {
namespace dmma {

constexpr int K = 64;            // the panel width: the inner dimension of every product here
constexpr int kPad = 68;         // shared row stride in doubles (68 = 4 mod 16: conflict-free fragments)
// A multiplier at least this large (or a NaN) means partial pivoting might have chosen another
// row at that column: the panel is refactored with explicit pivoting.  The margin below 1
// sends near-ties to the exact getf2 order as well.
constexpr double kMultLimit = 1.0 - 1e-12;

__device__ __forceinline__ void mma16x8x8(double (&c)[4], const double (&a)[4], const double (&b)[2])
{
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Copy BYTES (8 or 16) from global to shared; zero-fill when !valid (src is then not read).
template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src, bool valid)
{
    const uint32_t d = smem_addr(dst);
    const uint32_t n = valid ? BYTES : 0;
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// 64 x COLS block at (row0, col0) into sm[64][kPad] (columns past col_end read as zero).
template <int COLS, bool VEC, int NTHR>
__device__ __forceinline__ void stage_cols(double* sm, const double* __restrict__ g, uint32_t ld, uint32_t row0,
                                           uint32_t col0, uint32_t col_end, uint32_t tid = threadIdx.x)
{
    constexpr int PER = VEC ? 2 : 1;
    constexpr int CHUNKS = COLS / PER;
    for (uint32_t e = tid; e < (uint32_t)(K * CHUNKS); e += NTHR) {
        const uint32_t r = e / CHUNKS, c = (e % CHUNKS) * PER;
        const bool ok = col0 + c < col_end;  // (VEC: an odd col_end takes the row's padding along)
        const double* src = ok ? g + (size_t)(row0 + r) * ld + col0 + c : g;
        cp_async<8 * PER>(sm + r * kPad + c, src, ok);
    }
}

// ---------------------------------------------------------------- pipelined trailing update
// C -= A B over a run of 64 x 64 tiles of one M x N block C (rows row0.., columns col0..),
// A: the 64 columns a_col.. of C's rows, B: the 64 rows b_row.. of C's columns.  Tiles in
// column-major order, so that consecutive tiles of a run share their B block.  One CTA of
// kUpdWarps warps (8: warp tile 32 x 16; 4: 32 x 32) per SM.  The C and A blocks of each tile
// stream into a two-deep ring of shared memory by cp.async, issued one whole tile ahead: while
// tile t is multiplied, tile t + 1's blocks are already there and tile t + 2's are in flight;
// the accumulators start from -C (shared memory) and the result goes from registers to global
// memory.  So every tile costs its MMAs, two barriers and a few shared loads, and the HBM
// traffic (C in and out) runs underneath.
#ifndef PVL_UPD_WARPS
#define PVL_UPD_WARPS 8
#endif
constexpr int kUpdTile = 64;
constexpr int kUpdWarps = PVL_UPD_WARPS;
constexpr int kUpdThreads = 32 * kUpdWarps;
static_assert(kUpdWarps == 4 || kUpdWarps == 8, "2 x 2 or 2 x 4 warps over a 64 x 64 tile");
struct UpdSmem {
    double a[2][kUpdTile * kPad];
    double c[2][kUpdTile * kPad];
    double b[K * kPad];
};

// ROWS x COLS block at (row0, col0) of a row-major matrix into sm[ROWS][kPad]; rows past
// row_end and columns past col_end are not copied (their contents are never used).
template <int ROWS, int COLS, bool VEC, int NTHR>
__device__ __forceinline__ void stage_tile(double* sm, const double* __restrict__ g, uint32_t ld, uint32_t row0,
                                           uint32_t row_end, uint32_t col0, uint32_t col_end, uint32_t tid)
{
    constexpr int PER = VEC ? 2 : 1;
    constexpr int CHUNKS = COLS / PER;
    for (uint32_t e = tid; e < (uint32_t)(ROWS * CHUNKS); e += NTHR) {
        const uint32_t r = e / CHUNKS, c = (e % CHUNKS) * PER;
        if (row0 + r < row_end && col0 + c < col_end)  // (VEC: an odd col_end takes the row's padding along)
            cp_async<8 * PER>(sm + r * kPad + c, g + (size_t)(row0 + r) * ld + col0 + c, true);
    }
}

template <bool VEC>
__device__ __forceinline__ void update_tiles(UpdSmem& s, double* __restrict__ Cm, uint32_t ld, uint32_t row0,
                                             uint32_t col0, uint32_t m, uint32_t nn, uint32_t a_col, uint32_t b_row,
                                             uint32_t t_begin, uint32_t t_end)
{
    constexpr int WN = kUpdWarps / 2;     // warps along N
    constexpr int MT = 2, NT = 8 / WN;    // warp tile 32 x (64 / WN)
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t g = lane >> 2, t4 = lane & 3;
    const uint32_t wm0 = (warp / WN) * 32, wn0 = (warp % WN) * (8 * NT);
    const uint32_t tiles_i = (m + kUpdTile - 1) / kUpdTile;
    if (t_begin >= t_end)
        return;
    auto coords = [&](uint32_t t, uint32_t& i0, uint32_t& j0, uint32_t& me, uint32_t& ne) {
        i0 = (t % tiles_i) * kUpdTile;
        j0 = (t / tiles_i) * kUpdTile;
        me = min((uint32_t)kUpdTile, m - i0);
        ne = min((uint32_t)kUpdTile, nn - j0);
    };
    // tile t's A block (rows of C, the panel's columns) and C block into ring slot `buf`
    auto stage_ac = [&](uint32_t t, int buf) {
        uint32_t i0, j0, me, ne;
        coords(t, i0, j0, me, ne);
        stage_tile<kUpdTile, K, VEC, kUpdThreads>(s.a[buf], Cm, ld, row0 + i0, row0 + i0 + me, a_col, a_col + K, tid);
        stage_tile<kUpdTile, kUpdTile, VEC, kUpdThreads>(s.c[buf], Cm, ld, row0 + i0, row0 + i0 + me, col0 + j0,
                                                         col0 + j0 + ne, tid);
    };
    auto stage_b = [&](uint32_t t) {
        uint32_t i0, j0, me, ne;
        coords(t, i0, j0, me, ne);
        stage_cols<kUpdTile, VEC, kUpdThreads>(s.b, Cm, ld, b_row, col0 + j0, col0 + j0 + ne, tid);
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    // prologue: {B, A/C of the first tile}, {A/C of the second} -- one commit group each
    stage_b(t_begin);
    stage_ac(t_begin, 0);
    commit();
    if (t_begin + 1 < t_end)
        stage_ac(t_begin + 1, 1);
    commit();
    bool b_new = false;  // the most recent group holds a new B block
    for (uint32_t t = t_begin; t < t_end; ++t) {
        const int cur = (int)((t - t_begin) & 1u);
        // this tile's group is the second most recent, unless the most recent one holds its B
        if (b_new)
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        else
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        uint32_t i0, j0, me, ne;
        coords(t, i0, j0, me, ne);
        double acc[MT][NT][4];
        const double* cs = s.c[cur];
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t row = wm0 + 16 * i + g + 8 * h, col = wn0 + 8 * j + 2 * t4;
                    const double2 v = *reinterpret_cast<const double2*>(cs + row * kPad + col);
                    acc[i][j][2 * h] = -v.x;  // rows / columns outside the block: never stored
                    acc[i][j][2 * h + 1] = -v.y;
                }
        const double* as = s.a[cur];
#pragma unroll
        for (int k0 = 0; k0 < K; k0 += 8) {
            double af[MT][4], bf[NT][2];
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                const double* p = as + (wm0 + 16 * i + g) * kPad + k0 + t4;
                af[i][0] = p[0];
                af[i][1] = p[8 * kPad];
                af[i][2] = p[4];
                af[i][3] = p[8 * kPad + 4];
            }
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const double* p = s.b + (k0 + t4) * kPad + wn0 + 8 * j + g;
                bf[j][0] = p[0];
                bf[j][1] = p[4 * kPad];
            }
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int j = 0; j < NT; ++j)
                    mma16x8x8(acc[i][j], af[i], bf[j]);
        }
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const uint32_t col = wn0 + 8 * j + 2 * t4;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t row = wm0 + 16 * i + g + 8 * h;
                    if (row >= me)
                        continue;
                    double* cp = Cm + (size_t)(row0 + i0 + row) * ld + col0 + j0 + col;
                    const double v0 = -acc[i][j][2 * h], v1 = -acc[i][j][2 * h + 1];
                    if (VEC && col + 1 < ne) {
                        *reinterpret_cast<double2*>(cp) = make_double2(v0, v1);
                    } else {
                        if (col < ne)
                            cp[0] = v0;
                        if (col + 1 < ne)
                            cp[1] = v1;
                    }
                }
            }
        __syncthreads();  // slot `cur` (and B, if the next tile starts a column) may be refilled
        b_new = t + 1 < t_end && (t + 1) / tiles_i != t / tiles_i;
        if (b_new)
            stage_b(t + 1);
        if (t + 2 < t_end)
            stage_ac(t + 2, cur);
        commit();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");  // nothing in flight when the CTA exits
}

}  // namespace dmma
}  // namespace pvl
