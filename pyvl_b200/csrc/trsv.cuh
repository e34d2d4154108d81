// Wavefront triangular solve over 64-row blocks (the solve half of pvl_lu_solve).
//
// One CTA per row block, all co-resident (cooperative launch).  LOWER: unit-lower forward
// substitution, block b needs x of blocks 0..b-1; UPPER: backward substitution, block b needs
// x of blocks nblk-1..b+1.
//
// The solution values are their own ready flags: x starts as all-ones bit patterns (kNotReady, a
// NaN that no stored value has -- a result with those bits is stored as the canonical NaN), a
// block stores its 64 values with plain 8-byte stores, and the blocks that need them poll the
// values themselves.  So the chain from one block to the next is one store, one L2 read, a
// barrier and two 64 x 64 products from registers, without a fence, a flag and a second read.
// It is what bounds the solve, not the 134 MB of factors (20 us): 2 n / 64 links at 1.3-1.6 us,
// measured n = 1024: 51 us, 4096: 209 us, 5120: 274 us; with a flag per block, polled before the
// values were read, 2.8 us (107, 361 and 440 us).
// Thread (r, q) = (tid / 4, tid % 4) takes row r, columns q + 4 i, of every 64 x 64 block, so a
// row's sum is 16 FMAs and two shuffles.  Its entries of the blocks to come travel by cp.async
// through slots of its own in a three-stage ring of shared memory, two blocks ahead of the
// dependency awaited (a block arrives from memory in about the time of one link); its entries
// of the inverted diagonal block wait in registers.
//
// Waits are bounded: a thread that has polled `spin_limit` times sets *err, and its block stores
// NaNs (so that no later block waits on it in vain) and ends; the solution is then invalid and
// the caller reports PVL_ERR_TIMEOUT.  `skip_block` (normally -1) names a block that returns at
// once without storing anything: only a test uses it, to make the waits of every later block
// run out.
#pragma once

#include <cstdint>

#include "dmma.cuh"

namespace pvl {
namespace trsv {

constexpr int kRB = 64;         // rows per block (the LU's panel width)
constexpr int kThreads = 256;   // 64 rows x 4 threads
constexpr long long kSpinLimit = 5000000;  // ~2 s at ~0.4 us per poll
constexpr int kStages = 3;
constexpr size_t kSmem = (size_t)kStages * 16 * kThreads * sizeof(double);  // two CTAs per SM
constexpr unsigned long long kNotReady = ~0ull;
constexpr int kNotReadyByte = 0xFF;  // cudaMemset value of an unsolved x

__device__ __forceinline__ unsigned long long ld_value(const double* p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_value(double* p, double v)
{
    unsigned long long b = (unsigned long long)__double_as_longlong(v);
    if (b == kNotReady)
        b = 0x7FF8000000000000ull;
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(b) : "memory");
}

// M: the LU factors (row-major, lda); inv: the inverted diagonal blocks, (nblk, 2, 64, 64) with
// [b][0] = L_bb^-1 and [b][1] = U_bb^-1 (a partial last block padded with identity).  Right-hand
// side rhs[perm[i]] (rhs[i] without perm); x: the solution, kNotReady everywhere on entry; out (may
// be NULL, or rhs when perm is NULL): a second copy of it; flags (may be NULL): flags[b] = 1 when
// block b is done.
template <bool LOWER>
__global__ void __launch_bounds__(kThreads, 2) wavefront_kernel(uint32_t n, const double* __restrict__ M, uint32_t lda,
                                                                const double* __restrict__ inv, const double* rhs,
                                                                const int32_t* __restrict__ perm, double* x,
                                                                double* out, int32_t* flags, int32_t* err,
                                                                long long spin_limit, int32_t skip_block)
{
    extern __shared__ __align__(16) double s_ring[];  // [stage][i][thread]
    __shared__ double s_x[2][kRB];
    __shared__ double s_r[kRB];
    __shared__ int s_abort;
    const uint32_t nblk = (n + kRB - 1) / kRB;
    const uint32_t b = LOWER ? blockIdx.x : nblk - 1 - blockIdx.x;
    if ((int32_t)b == skip_block)
        return;
    const uint32_t r0 = b * kRB, rows = min((uint32_t)kRB, n - r0);
    const uint32_t r = threadIdx.x >> 2, q = threadIdx.x & 3;
    const uint32_t n_dep = LOWER ? b : nblk - 1 - b;
    auto dep = [&](uint32_t step) { return (LOWER ? step : nblk - 1 - step) * kRB; };  // its first row
    double dinv[16], part[4] = {0.0, 0.0, 0.0, 0.0};
    double* slot = s_ring + threadIdx.x;
    auto load_block = [&](uint32_t step) {  // one commit group per step, empty past the last
        if (step < n_dep) {
            const uint32_t c0 = dep(step);
            const double* mrow = M + (size_t)(r0 + r) * lda + c0;
            double* dst = slot + (size_t)(step % kStages) * 16 * kThreads;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const uint32_t c = q + 4 * i;
                const bool ok = r < rows && c0 + c < n;
                dmma::cp_async<8>(dst + i * kThreads, ok ? mrow + c : M, ok);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the value of x that this thread (of the first 64) waits for at a step
    auto peek = [&](uint32_t c0) {
        return threadIdx.x < kRB && c0 + threadIdx.x < n ? ld_value(x + c0 + threadIdx.x) : 0ull;
    };
    unsigned long long v = 0ull;
    load_block(0);
    load_block(1);
    if (n_dep > 0)
        v = peek(dep(0));
    const double* D = inv + ((size_t)b * 2 + (LOWER ? 0 : 1)) * kRB * kRB + r * kRB + q;
#pragma unroll
    for (int i = 0; i < 16; ++i)
        dinv[i] = D[4 * i];
    const double own = r < rows && q == 0 ? rhs[perm ? (size_t)perm[r0 + r] : (size_t)(r0 + r)] : 0.0;
    if (threadIdx.x == 0)
        s_abort = 0;
    __syncthreads();
    for (uint32_t step = 0; step < n_dep; ++step) {
        if (threadIdx.x < kRB) {
            const uint32_t c0 = dep(step);
            long long spins = 0;
            while (v == kNotReady) {
                v = ld_value(x + c0 + threadIdx.x);
                if (++spins > spin_limit) {
                    atomicExch(err, 1);
                    s_abort = 1;
                    break;
                }
            }
            s_x[step & 1][threadIdx.x] = __longlong_as_double((long long)v);
        }
        __syncthreads();
        if (s_abort) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            if (q == 0 && r < rows)
                st_value(x + r0 + r, __longlong_as_double(0x7FF8000000000000ll));
            if (threadIdx.x == 0 && flags)
                flags[b] = 1;
            return;
        }
        load_block(step + 2);  // overwrites the slots read in the previous step, by this thread alone
        if (step + 1 < n_dep)
            v = peek(dep(step + 1));
        asm volatile("cp.async.wait_group 2;" ::: "memory");
        const double* xs = s_x[step & 1];
        const double* m = slot + (size_t)(step % kStages) * 16 * kThreads;
#pragma unroll
        for (int i = 0; i < 16; ++i)
            part[i & 3] = fma(m[i * kThreads], xs[q + 4 * i], part[i & 3]);
    }
    // x_b = inv(D_bb) (rhs_b - sums)
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    double s = (part[0] + part[1]) + (part[2] + part[3]);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (q == 0)
        s_r[r] = own - s;
    __syncthreads();
    double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int i = 0; i < 16; ++i)
        t[i & 3] = fma(dinv[i], s_r[q + 4 * i], t[i & 3]);
    s = (t[0] + t[1]) + (t[2] + t[3]);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (q == 0 && r < rows) {
        st_value(x + r0 + r, s);
        if (out)
            out[r0 + r] = s;
    }
    if (flags) {
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0)
            flags[b] = 1;
    }
}

}  // namespace trsv
}  // namespace pvl
