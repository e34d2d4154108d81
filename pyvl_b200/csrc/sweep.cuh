// Pair arithmetic of the FP64 N-body sweep (line_sum_f64_kernel), sm_100a.
//
// The quantities of segment_induction (pvl_common.cuh) in Pluecker form about an origin o
// that the CTA chooses (the centroid of its points): a segment is staged once per CTA as
//   d (unit direction), m = (r1 - o) x d, e = d . (r1 - o), len, gamma len, gamma
// (80 bytes, five 16-byte shared loads per pair; gamma is read only by the near pairs), and
// for a point p' = p - o
//   t1 = d . p' - e = d . (p - r1),   c = p' x d - m = (p - r1) x d
// from 9 FMAs instead of 3 differences and 9 products per pair.  Rounding is relative to
// |p - o| + |r1 - o| instead of |p - r1|; the points of one CTA are neighbours (ring or
// wake-node order, or one case of a batch), so |p - o| stays of the order of the body.
// Everything after c and t1 -- h^2, x = h^2 + t1 t2, the far-field series with the Newton
// reciprocal, the atan2 form for near pairs, the cut-off -- is segment_induction's, scaled by gamma,
// with w = h^2 len^2 / x^2 formed as h^2 (len / x)^2.
#pragma once

#include <cstdint>

#include "pvl_common.cuh"

namespace pvl {

struct __align__(16) SweepSeg {
    double dx, dy, dz, mx, my, mz, e, len, glen, gamma;
};

struct SweepGeo {
    double cx, cy, cz, hsq, x, r, w;
};

// The segment g about origin o (o[0..2], usually in shared memory).
__device__ __forceinline__ SweepSeg sweep_seg(const Segment<double>& g, const double* o)
{
    const double rx = g.r1x - o[0], ry = g.r1y - o[1], rz = g.r1z - o[2];
    SweepSeg t;
    t.dx = g.dx;
    t.dy = g.dy;
    t.dz = g.dz;
    t.mx = ry * g.dz - rz * g.dy;
    t.my = rz * g.dx - rx * g.dz;
    t.mz = rx * g.dy - ry * g.dx;
    t.e = g.dx * rx + g.dy * ry + g.dz * rz;
    t.len = g.len;
    t.glen = g.glen;
    t.gamma = g.gamma;
    return t;
}

__device__ __forceinline__ SweepGeo sweep_geo(const SweepSeg& s, double px, double py, double pz)
{
    SweepGeo g;
    const double t1 = fma(s.dz, pz, fma(s.dy, py, fma(s.dx, px, -s.e)));
    g.cx = fma(py, s.dz, -fma(pz, s.dy, s.mx));
    g.cy = fma(pz, s.dx, -fma(px, s.dz, s.my));
    g.cz = fma(px, s.dy, -fma(py, s.dx, s.mz));
    g.hsq = g.cx * g.cx + g.cy * g.cy + g.cz * g.cz;
    g.x = g.hsq + t1 * (t1 - s.len);
    g.r = FarSeries<double>::rcp(g.x);
    const double a = s.len * g.r;
    g.w = g.hsq * (a * a);
    return g;
}

// Far pairs by the arctangent series (selected, no branch), the rare near pairs by atan2 in a
// branch, pairs inside the cut-off skipped; gamma_k u_k(p) added to acc.
__device__ __forceinline__ void sweep_add(const SweepSeg& s, const SweepGeo& g, double tol2, Vec3<double>& acc)
{
    const bool ok = !lt_nn(g.hsq, tol2);
    const bool far = ok && pos_hi(g.x) && le_hi(g.w, FarSeries<double>::kW);
    double mag = far ? -s.glen * g.r * FarSeries<double>::sum(g.w) : 0.0;
    if (ok && !far) {
        const double rh = rsqrt(g.hsq);
        const double h = g.hsq * rh;
        mag = s.gamma * atan2(-h * s.len, g.x) * rh;
    }
    acc.x += g.cx * mag;
    acc.y += g.cy * mag;
    acc.z += g.cz * mag;
}

// gamma_a u_a(p_a) and gamma_b u_b(p_b) added to A and B (one accumulator, or two points'): as two
// sweep_add calls, with the tier of both pairs of all lanes decided by one vote, so that the usual
// eight or four terms run without a branch per pair.  Every lane of the warp calls it.  The batched
// sweep gains (64 wings: 1853 -> 1761 us); line_sum_f64_kernel, with nine tenths of the registers
// that this form asks for at its occupancy, does not (461 us either way) and keeps sweep_add.
__device__ __forceinline__ void sweep_add2(const SweepSeg& a, const SweepGeo& ga, const SweepSeg& b,
                                           const SweepGeo& gb, double tol2, Vec3<double>& A, Vec3<double>& B)
{
    using F = FarSeries<double>;
    const bool cut_a = lt_nn(ga.hsq, tol2), cut_b = lt_nn(gb.hsq, tol2);
    const int ma = cut_a ? 0 : pos_hi(ga.x) ? hi32(ga.w) : 0x7FFFFFFF;
    const int mb = cut_b ? 0 : pos_hi(gb.x) ? hi32(gb.w) : 0x7FFFFFFF;
    const int worst = max(ma, mb);
    if (__any_sync(0xFFFFFFFFu, worst > hi32(0.01))) {
        sweep_add(a, ga, tol2, A);
        sweep_add(b, gb, tol2, B);
        return;
    }
    double fa = -a.glen * ga.r, fb = -b.glen * gb.r;
    if (__any_sync(0xFFFFFFFFu, worst > hi32(1e-4))) {
        fa *= F::sum_tier<8>(ga.w);
        fb *= F::sum_tier<8>(gb.w);
    } else {
        fa *= F::sum_tier<4>(ga.w);
        fb *= F::sum_tier<4>(gb.w);
    }
    fa = cut_a ? 0.0 : fa;
    fb = cut_b ? 0.0 : fb;
    A.x += ga.cx * fa;
    A.y += ga.cy * fa;
    A.z += ga.cz * fa;
    B.x += gb.cx * fb;
    B.y += gb.cy * fb;
    B.z += gb.cz * fb;
}

// o = centroid of the CTA's valid points (0 if none), in fixed summation order, from each
// thread's sum of its valid points (sx, sy, sz) and their count n; every thread of the CTA
// must call it.  red: THREADS / 32 x 4 doubles of shared memory, o: 3.
template <int THREADS>
__device__ __forceinline__ void cta_centroid(double sx, double sy, double sz, double n, double (*red)[4], double* o)
{
    double v[4] = {sx, sy, sz, n};
#pragma unroll
    for (int c = 0; c < 4; ++c)
        for (int k = 16; k > 0; k >>= 1)
            v[c] += __shfl_xor_sync(0xffffffffu, v[c], k);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int c = 0; c < 4; ++c)
            red[threadIdx.x >> 5][c] = v[c];
    __syncthreads();
    if (threadIdx.x < 3) {
        double t = 0.0, n = 0.0;
        for (int w = 0; w < THREADS / 32; ++w) {
            t += red[w][threadIdx.x];
            n += red[w][3];
        }
        o[threadIdx.x] = n > 0.0 ? t / n : 0.0;
    }
    __syncthreads();
}

}  // namespace pvl
