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

// ---------------------------------------------------------------- pipelined trailing update
// C -= A B over a run of 64 x 64 tiles of one M x N block C (rows row0.., columns col0..),
// A: the 64 columns a_col.. of C's rows, B: the 64 rows b_row.. of C's columns.  Tiles in
// column-major order, so that consecutive tiles of a run share their B block.  A run belongs to a
// group of eight warps (warp tile 32 x 16, four independent MMAs per step), and a CTA holds two
// groups that share nothing but the SM: while one waits at its barriers, stores its tile or
// fetches, the other's MMAs keep the tensor pipe busy.  The A blocks stream into the group's
// two-deep ring by cp.async, one tile ahead; C goes from global memory to registers while the
// tile is multiplied (the product is formed by itself and subtracted at the end) and back, and the
// next tile's C is prefetched into L2 meanwhile.  What each part gave to the factorisation of 4096
// (when the rest of it took 0.2 ms more than now): one group of eight warps per CTA with C in the ring
// 3323 us, two groups of four warps 3243, two of eight 3167 (four warps per scheduler hide the
// fragment loads), with the prefetch 3140.  The first update of n = 4096, 3968 x 3968: 96 us, the
// FP64 tensor pipe active 66 % of it; a 4032 x 4032 one on 133 SMs took 106 us, 82 with C's traffic
// left out and 69 with the MMAs left out (which need 66 at the pipe's rate): the two overlap only in
// part.
constexpr int kUpdTile = 64;
constexpr int kUpdGroups = 2;  // (update_tiles names one barrier for each)
constexpr int kUpdGroupThreads = 256;
constexpr int kUpdThreads = kUpdGroups * kUpdGroupThreads;
struct UpdSmem {
    double a[2][kUpdTile * kPad];
    double b[K * kPad];
};

// C of one warp-tile entry pair; issued before the MMAs (volatile keeps it there).
__device__ __forceinline__ double2 load_c2(const double* p)
{
    double2 v;
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ double load_c1(const double* p)
{
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

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

// `group`: which group of the CTA this is (named barrier 1 + group), tid: thread of the group.
template <bool VEC>
__device__ __forceinline__ void update_tiles(UpdSmem& s, int group, uint32_t tid, double* __restrict__ Cm, uint32_t ld,
                                             uint32_t row0, uint32_t col0, uint32_t m, uint32_t nn, uint32_t a_col,
                                             uint32_t b_row, uint32_t t_begin, uint32_t t_end)
{
    constexpr int WN = kUpdGroupThreads / 64, MT = 2, NT = 8 / WN;  // 2 x WN warps, warp tile 32 x (64 / WN)
    const uint32_t lane = tid & 31, warp = tid >> 5;
    const uint32_t g = lane >> 2, t4 = lane & 3;
    const uint32_t wm0 = (warp / WN) * 32, wn0 = (warp % WN) * (8 * NT);
    const uint32_t tiles_i = (m + kUpdTile - 1) / kUpdTile;
    if (t_begin >= t_end)
        return;
    auto barrier = [&] {  // constant names: the CTA then holds three barriers, not all sixteen
        if (group == 0)
            asm volatile("bar.sync 1, %0;" ::"n"(kUpdGroupThreads) : "memory");
        else
            asm volatile("bar.sync 2, %0;" ::"n"(kUpdGroupThreads) : "memory");
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    uint32_t ti = t_begin % tiles_i, tj = t_begin / tiles_i;  // tile t's row and column of tiles
    auto stage_a = [&](uint32_t i, int buf) {
        const uint32_t i0 = i * kUpdTile;
        stage_tile<kUpdTile, K, VEC, kUpdGroupThreads>(s.a[buf], Cm, ld, row0 + i0, row0 + min(m, i0 + kUpdTile), a_col,
                                                       a_col + K, tid);
    };
    auto stage_b = [&](uint32_t j) {
        const uint32_t j0 = j * kUpdTile;
        stage_tile<K, kUpdTile, VEC, kUpdGroupThreads>(s.b, Cm, ld, b_row, b_row + K, col0 + j0,
                                                       col0 + min(nn, j0 + kUpdTile), tid);
    };
    // prologue: {B and A of the first tile}, {A of the second} -- one commit group each
    stage_b(tj);
    stage_a(ti, 0);
    commit();
    if (t_begin + 1 < t_end)
        stage_a(ti + 1 == tiles_i ? 0 : ti + 1, 1);
    commit();
    // the C block of tile (i, j) into L2: 64 rows of four 128-byte lines
    auto prefetch_c = [&](uint32_t i, uint32_t j) {
        for (uint32_t e = tid; e < 4u * kUpdTile; e += kUpdGroupThreads) {
            const uint32_t r = i * kUpdTile + e / 4, c = j * kUpdTile + (e % 4) * 16;
            if (r < m && c < nn)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(Cm + (size_t)(row0 + r) * ld + col0 + c));
        }
    };
    bool b_new = false;  // the most recent group holds a new B block
    for (uint32_t t = t_begin; t < t_end; ++t) {
        const int cur = (int)((t - t_begin) & 1u);
        const uint32_t i0 = ti * kUpdTile, j0 = tj * kUpdTile;
        const uint32_t me = min((uint32_t)kUpdTile, m - i0), ne = min((uint32_t)kUpdTile, nn - j0);
        double* const cw = Cm + (size_t)(row0 + i0 + wm0 + g) * ld + col0 + j0 + wn0 + 2 * t4;
        // C of this warp's 32 x 16 (32 x 8 NT): entry h of (i, j) is row wm0 + 16 i + 8 h + g
        double2 c[MT][NT][2];
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const bool row_ok = wm0 + 16 * i + 8 * h + g < me;
                const double* cp = cw + (size_t)(16 * i + 8 * h) * ld;
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const uint32_t col = wn0 + 8 * j + 2 * t4;
                    c[i][j][h] = make_double2(0.0, 0.0);
                    if (VEC) {
                        if (row_ok && col < ne)  // (an odd ne takes the row's padding along)
                            c[i][j][h] = load_c2(cp + 8 * j);
                    } else {
                        if (row_ok && col < ne)
                            c[i][j][h].x = load_c1(cp + 8 * j);
                        if (row_ok && col + 1 < ne)
                            c[i][j][h].y = load_c1(cp + 8 * j + 1);
                    }
                }
            }
        const uint32_t ni = ti + 1 == tiles_i ? 0 : ti + 1, nj = ni ? tj : tj + 1;
        if (t + 1 < t_end)
            prefetch_c(ni, nj);
        // this tile's blocks are in the second most recent group, unless the most recent one holds its B
        if (b_new)
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        else
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        barrier();
        double acc[MT][NT][4];
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    acc[i][j][e] = 0.0;
        const double* ap = s.a[cur] + (wm0 + g) * kPad + t4;
        const double* bp = s.b + t4 * kPad + wn0 + g;
#pragma unroll 4
        for (int k0 = 0; k0 < K; k0 += 8, ap += 8, bp += 8 * kPad) {
            double af[MT][4], bf[NT][2];
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                af[i][0] = ap[16 * i * kPad];
                af[i][1] = ap[(16 * i + 8) * kPad];
                af[i][2] = ap[16 * i * kPad + 4];
                af[i][3] = ap[(16 * i + 8) * kPad + 4];
            }
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                bf[j][0] = bp[8 * j];
                bf[j][1] = bp[4 * kPad + 8 * j];
            }
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int j = 0; j < NT; ++j)
                    mma16x8x8(acc[i][j], af[i], bf[j]);
        }
        barrier();  // ring slot `cur` (and B, if the next tile starts a column) may be refilled
        b_new = t + 1 < t_end && nj != tj;
        if (b_new)
            stage_b(nj);
        if (t + 2 < t_end)
            stage_a(ni + 1 == tiles_i ? 0 : ni + 1, cur);
        commit();
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const bool row_ok = wm0 + 16 * i + 8 * h + g < me;
                double* cp = cw + (size_t)(16 * i + 8 * h) * ld;
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const uint32_t col = wn0 + 8 * j + 2 * t4;
                    const double v0 = c[i][j][h].x - acc[i][j][2 * h], v1 = c[i][j][h].y - acc[i][j][2 * h + 1];
                    if (VEC && row_ok && col + 1 < ne) {
                        *reinterpret_cast<double2*>(cp + 8 * j) = make_double2(v0, v1);
                    } else {
                        if (row_ok && col < ne)
                            cp[8 * j] = v0;
                        if (row_ok && col + 1 < ne)
                            cp[8 * j + 1] = v1;
                    }
                }
            }
        ti = ni;
        tj = nj;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");  // nothing in flight when the group ends
}

}  // namespace dmma
}  // namespace pvl
