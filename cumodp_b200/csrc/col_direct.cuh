// Column passes of 2^1 .. 2^10 rows with the operands in registers.
//
// Level 0 of the forward pass reads its words straight from global memory (a
// task owns rows o + R1 m of one column), the last level stores straight to
// global memory, and shared memory is only the exchange between the two
// levels; up to 2^5 rows one level is the whole column and there is no
// exchange at all.  The inverse pass is the transposed sequence.  One tile
// per CTA, 1024 threads of 64 registers per SM (two CTAs for 2^10 rows: one
// loads while the other computes).  The pipelined kernels this replaces
// staged every tile through shared memory by cp.async, half or a whole tile
// ahead, on 16 warps per SM.
// Rows leave the forward pass and enter the inverse one in bit-reversed order
// of the frequency, for every split into levels.
// Bound by integer issue and the strided accesses' latency.  Measured on B200
// (2^24 words, one launch between events): 2^10 rows, two half-empty operands
// 79 -> 68 us, one full operand 51 -> 44, inverse 43 -> 40; a batch of 4096
// uneven products (columns of 2^3-2^6 rows) 1119 -> 1025 us.  8-column tiles of
// 256 threads for 2^10 rows were slower (the 2^24-point product 260 us for 252).
#pragma once
#include "large_product.cuh"

namespace cmb {

constexpr int kMaxDirectColLog = 10;

__host__ __device__ constexpr bool cold_two(int l1) { return l1 > 5; }
__host__ __device__ constexpr int cold_r0(int l1) { return cold_two(l1) ? 1 << col_plan(l1).logr[0] : 1 << l1; }
__host__ __device__ constexpr int cold_r1(int l1) { return (1 << l1) / cold_r0(l1); }
// Columns of a tile: one per lane, or half a warp's where a tile of 2^10 rows fills 64 KiB.
__host__ __device__ constexpr int cold_cols(int l1) { return !cold_two(l1) ? 128 : l1 == 10 ? 16 : 32; }
__host__ __device__ constexpr int cold_threads(int l1) { return !cold_two(l1) ? 128 : l1 <= 7 ? 256 : 512; }
__host__ __device__ constexpr int cold_ctas(int l1) { return 1024 / cold_threads(l1); }
// Words between the R1-row blocks of a tile: with 16 columns a half-warp holds
// one block's row, and a 16-word pad puts the other half-warp's block into the
// other banks.
__host__ __device__ constexpr int cold_block(int l1) { return cold_r1(l1) * cold_cols(l1) + (cold_cols(l1) == 16 ? 16 : 0); }
__host__ __device__ constexpr size_t cold_smem(int l1) {
    return cold_two(l1) ? (size_t)cold_r0(l1) * cold_block(l1) * sizeof(u32) : 0;
}

#ifdef __CUDACC__

// Shoup twiddles 2 k and 2 k + 1 of a task.
__device__ __forceinline__ uint4 cold_tw2(const Tw* __restrict__ t, int k) {
    return __ldg(reinterpret_cast<const uint4*>(t) + k);
}

// Pass A; grid (n2 / columns, operands, jobs).
template <int L1>
__global__ void __launch_bounds__(cold_threads(L1), cold_ctas(L1)) k_cold_fwd(const __grid_constant__ LargeArgs A) {
    constexpr bool TWO = cold_two(L1);
    constexpr int R0 = cold_r0(L1), R1 = cold_r1(L1), TC = cold_cols(L1), T = cold_threads(L1), BL = cold_block(L1);
    extern __shared__ __align__(16) u32 tile[];
    const LargeJob& J = A.jobs ? A.jobs[blockIdx.z] : A.job0;
    const bool second = blockIdx.y != 0;
    const u32* src = second ? J.b : J.a;
    const int len = second ? J.lb : J.la;
    u32* dst = second ? J.wb : J.wa;
    const int n2 = 1 << A.l2, c = threadIdx.x % TC, col = blockIdx.x * TC + c;
    const u32 p = A.pkc.p, p2 = A.pkc.p2, oneq = A.pkc.one_q;
    if (!TWO && col >= n2) return;
    const bool full = len > (n2 << L1) / 2;  // else the upper half of the rows is padding
    for (int o = threadIdx.x / TC; o < R1; o += T / TC) {
        u32 x[R0];
        int gi = o * n2 + col;
        const u32* g = src + gi;
        const int step = R1 * n2;
#pragma unroll
        for (int m = 0; m < R0 / 2; ++m, gi += step, g += step) x[m] = gi < len ? __ldg(g) : 0u;
        if (!full) {
            dif_regs_halfzero<R0, TWO>(x, A.pkc.rc.f, p, p2, oneq);
        } else {
#pragma unroll
            for (int m = R0 / 2; m < R0; ++m, gi += step, g += step) x[m] = gi < len ? __ldg(g) : 0u;
#pragma unroll
            for (int m = 0; m < R0; ++m) x[m] = mul_shoup(x[m], 1u, oneq, p);
            dif_regs<R0, TWO>(x, A.pkc.rc.f, p, p2);
        }
        if constexpr (TWO) {
            const Tw* t = A.twc + o * R0;
            u32* s = tile + o * TC + c;
            s[0] = x[0];
#pragma unroll
            for (int k = 0; k < R0 / 2; ++k) {
                const uint4 w = cold_tw2(t, k);
                if (k > 0) s[2 * k * BL] = mul_shoup(x[2 * k], w.x, w.y, p);
                s[(2 * k + 1) * BL] = mul_shoup(x[2 * k + 1], w.z, w.w, p);
            }
        } else {
            u32* out = dst + col;
#pragma unroll
            for (int m = 0; m < R0; ++m, out += n2) *out = x[m];
        }
    }
    if constexpr (TWO) {
        __syncthreads();
        for (int b = threadIdx.x / TC; b < R0; b += T / TC) {
            u32 x[R1];
            const u32* s = tile + b * BL + c;
#pragma unroll
            for (int m = 0; m < R1; ++m) x[m] = s[m * TC];
            dif_regs<R1>(x, A.pkc.rc.f, p, p2);
            u32* out = dst + (size_t)(b * R1) * n2 + col;
#pragma unroll
            for (int m = 0; m < R1; ++m, out += n2) *out = x[m];
        }
    }
}

// Pass C; grid (n2 / columns, 1, jobs).
template <int L1>
__global__ void __launch_bounds__(cold_threads(L1), cold_ctas(L1)) k_cold_inv(const __grid_constant__ LargeArgs A) {
    constexpr bool TWO = cold_two(L1);
    constexpr int R0 = cold_r0(L1), R1 = cold_r1(L1), TC = cold_cols(L1), T = cold_threads(L1), BL = cold_block(L1);
    extern __shared__ __align__(16) u32 tile[];
    const LargeJob& J = A.jobs ? A.jobs[blockIdx.z] : A.job0;
    const int n2 = 1 << A.l2, c = threadIdx.x % TC, col = blockIdx.x * TC + c, lh = J.lh;
    const u32 p = A.pkc.p, p2 = A.pkc.p2;
    if (!TWO && col >= n2) return;
    pdl_wait();  // pass B's output
    if constexpr (TWO) {
        for (int b = threadIdx.x / TC; b < R0; b += T / TC) {
            u32 x[R1];
            const u32* g = J.wa + (size_t)(b * R1) * n2 + col;
#pragma unroll
            for (int m = 0; m < R1; ++m, g += n2) x[m] = *g;
            dit_regs<R1>(x, A.pkc.rc.i, p, p2);
            u32* s = tile + b * BL + c;
#pragma unroll
            for (int m = 0; m < R1; ++m) s[m * TC] = x[m];
        }
        __syncthreads();
    }
    for (int o = threadIdx.x / TC; o < R1; o += T / TC) {
        u32 x[R0];
        if constexpr (TWO) {
            const Tw* t = A.twc + A.twc_inv + o * R0;
            const u32* s = tile + o * TC + c;
            x[0] = s[0];
#pragma unroll
            for (int k = 0; k < R0 / 2; ++k) {
                const uint4 w = cold_tw2(t, k);
                if (k > 0) x[2 * k] = mul_shoup(s[2 * k * BL], w.x, w.y, p);
                x[2 * k + 1] = mul_shoup(s[(2 * k + 1) * BL], w.z, w.w, p);
            }
        } else {
            const u32* g = J.wa + col;
#pragma unroll
            for (int m = 0; m < R0; ++m, g += n2) x[m] = *g;
        }
        dit_regs<R0, TWO>(x, A.pkc.rc.i, p, p2);
        int gi = o * n2 + col;
        const int step = R1 * n2;
        u32* out = J.h + gi;
#pragma unroll
        for (int m = 0; m < R0; ++m, gi += step, out += step)
            if (gi < lh) *out = red1(red2(x[m], p2), p);
    }
}

#endif  // __CUDACC__

}  // namespace cmb
