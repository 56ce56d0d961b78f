// Natural-order transforms of rows of 2^6 .. 2^14 words: independent ones, and
// those of a four-step transform.
//
// A row takes two or three levels of radix 8..32, the fewest that fit a
// thread's registers: level 0 reads its words straight from global memory (task
// o owns words o + TB m), the last level stores its outputs straight to global
// memory, and shared memory is only the exchange between levels.  A level's
// output k goes to digit k of the frequency (f = k0 + R0 k1 + R0 R1 k2: the
// bit reversal of a register DFT is a renaming of registers), so the last
// level's task (k0, k1) holds frequencies k0 + R0 k1 + R0 R1 k2: consecutive
// tasks are consecutive words, and natural order costs no pass.
// Bound by integer issue: two exchanges and one Shoup product per word and
// level boundary where the previous kernel ran four levels, a copy into shared memory
// before them and a reorder through it after them.  Measured on B200, 2^25
// words of rows, before -> after:
//   2^6   390 -> 54 us    2^9   115 -> 70 us    2^12  109 -> 70 us
//   2^7   209 -> 66 us    2^10   82 -> 70 us    2^13  115 -> 73 us
//   2^8   129 -> 50 us    2^11   90 -> 66 us    2^14  134 -> 96 us
// (2^14: radix 32 at 64 registers on two CTAs per SM).
#pragma once
#include "large_product.cuh"

namespace cmb {

__host__ __device__ constexpr LevelPlan nat_plan(int logl) {
    switch (logl) {
        case 6: return LevelPlan{2, {3, 3}};
        case 7: return LevelPlan{2, {3, 4}};
        case 8: return LevelPlan{2, {4, 4}};
        case 9: return LevelPlan{3, {3, 3, 3}};
        case 10: return LevelPlan{3, {3, 3, 4}};
        case 11: return LevelPlan{3, {4, 3, 4}};
        case 12: return LevelPlan{3, {4, 4, 4}};
        case 13: return LevelPlan{3, {5, 4, 4}};
        case 14: return LevelPlan{3, {5, 5, 4}};
        default: return LevelPlan{0, {0}};
    }
}
// Twiddles of level 0 ([k0][o0]), then of level 1 ([k1][o1]) when there are three.
__host__ __device__ constexpr int nat_entries(int logl) {
    return (1 << logl) + (nat_plan(logl).nlev == 3 ? 1 << (logl - nat_plan(logl).logr[0]) : 0);
}
// Threads of one row (its level-0 tasks), rows and threads of a CTA.
__host__ __device__ constexpr int nat_row_threads(int logl) { return 1 << (logl - nat_plan(logl).logr[0]); }
__host__ __device__ constexpr int nat_rows(int logl) { return nat_row_threads(logl) >= 128 ? 1 : 128 / nat_row_threads(logl); }
__host__ __device__ constexpr int nat_threads(int logl) { return nat_rows(logl) * nat_row_threads(logl); }
// Words of shared memory between two k0 blocks: the last level's tasks step
// through k0, so an odd step puts consecutive tasks into different banks (two
// ways for rows of 2^10).  The middle level's warps cover two k0 blocks one bank
// apart: two ways in every access (four for 2^9), 2^20 conflicts in a 2^24-point
// transform's rows.
__host__ __device__ constexpr int nat_stride(int logl) { return nat_row_threads(logl) + 1; }
__host__ __device__ constexpr int nat_words(int logl) { return nat_stride(logl) << nat_plan(logl).logr[0]; }
__host__ __device__ constexpr size_t nat_smem(int logl) { return (size_t)nat_rows(logl) * nat_words(logl) * sizeof(u32); }
// CTAs per SM the kernel is compiled for: radix 32 needs up to 64 registers, radix 16 about 48.
__host__ __device__ constexpr int nat_ctas(int logl) { return nat_plan(logl).logr[0] == 5 ? 1024 / nat_threads(logl) : 1280 / nat_threads(logl); }

// rev_bits of a constant.
__host__ __device__ constexpr u32 rev_bits_c(u32 j, int r) {
    u32 v = 0;
    for (int i = 0; i < r; ++i) v |= ((j >> i) & 1u) << (r - 1 - i);
    return v;
}

struct RowNatArgs {
    PrimeK pk;
    const Tw* __restrict__ tw;  // nat_entries; the output scale is folded into level 0's
    const u32* src;             // row s at src + s n
    u32* dst;                   // row out(s) at dst + out(s) n (may be src when out(s) = s)
    u32 rows;
    int scaled;                 // level 0's k0 = 0 twiddles are not 1
    int l1;                     // > 0: rows are slots of a column pass of 2^l1, out(s) = its frequency
    LevelPlan colpl;
    const Tw* __restrict__ slot;  // SLOT: slot s's nat_slot_entries from s times that on
    long long job_stride;         // words between the transforms of grid row blockIdx.y
};
// Rows of a four-step transform (SLOT): word c of slot s is multiplied by the
// inter-pass twiddle W^c, W = w^k1(s).  Task o's words are c = o + TB m, so
// W^c = W^(TB m) W^o: the first is one of R0 factors of the slot, on the way
// in; the second is the task's own and commutes with the DFT.  Per slot: W^(TB
// m) for m < R0, then W^o for every task.
__host__ __device__ constexpr int nat_slot_entries(int logl) { return (1 << nat_plan(logl).logr[0]) + nat_row_threads(logl); }
// Exponent of entry t of nat_slot_tables' array to the base w.
struct SlotExponent {
    LevelPlan colpl;
    int l1, r0, tb;  // columns of 2^l1; level 0's radix and tasks
    __host__ __device__ u32 operator()(u32 t) const {
        const u32 s = t / (u32)(r0 + tb), i = t % (u32)(r0 + tb);
        return col_slot_to_k1(s, colpl, l1) * (i < (u32)r0 ? tb * i : i - r0);
    }
};

#ifdef __CUDACC__

template <int L2, bool SLOT>
__global__ void __launch_bounds__(nat_threads(L2), nat_ctas(L2)) k_row_nat(const __grid_constant__ RowNatArgs A) {
    constexpr LevelPlan PL = nat_plan(L2);
    constexpr bool THREE = PL.nlev == 3;
    constexpr int n = 1 << L2, TPR = nat_row_threads(L2), S = nat_stride(L2);
    constexpr int R0 = 1 << PL.logr[0], TB0 = n / R0;
    constexpr int R1 = THREE ? 1 << PL.logr[1] : 1, TB1 = TB0 / R1;  // three levels: level 1
    constexpr int RL = 1 << PL.logr[PL.nlev - 1];                    // the last level
    extern __shared__ __align__(16) u32 smem[];
    const int t = threadIdx.x % TPR, rl = threadIdx.x / TPR;
    const u32 s = blockIdx.x * nat_rows(L2) + rl;
    const bool has = s < A.rows;
    u32* const sm = smem + rl * nat_words(L2);
    const u32 p = A.pk.p, p2 = A.pk.p2;
    {
        u32 x[R0];
        const size_t job = SLOT ? blockIdx.y * (size_t)A.job_stride : 0;
        const u32* src = A.src + job + (size_t)(has ? s : 0) * n + t;
#pragma unroll
        for (int m = 0; m < R0; ++m) x[m] = src[TB0 * m];  // (may be the rows written below)
        uint2 wo = make_uint2(1u, 0u);
        if constexpr (SLOT) {  // a column pass's words, below 2p
            const uint2* f = reinterpret_cast<const uint2*>(A.slot + (size_t)(has ? s : 0) * nat_slot_entries(L2));
            wo = __ldg(f + R0 + t);
#pragma unroll
            for (int m = 1; m < R0; ++m) {
                const uint2 w = __ldg(f + m);
                x[m] = mul_shoup(x[m], w.x, w.y, p);
            }
        } else {
#pragma unroll
            for (int m = 0; m < R0; ++m) x[m] = mul_shoup(x[m], 1u, A.pk.one_q, p);
        }
        dif_regs<R0, true>(x, A.pk.rc.f, p, p2);
        const Tw* tw = A.tw + t;
#pragma unroll
        for (int j = 0; j < R0; ++j) {
            const int k = (int)rev_bits_c(j, PL.logr[0]);
            if (j > 0 || A.scaled) {
                const uint2 w = __ldg(reinterpret_cast<const uint2*>(tw + TB0 * k));
                x[j] = mul_shoup(x[j], w.x, w.y, p);
            }
            if constexpr (SLOT) x[j] = mul_shoup(x[j], wo.x, wo.y, p);
            sm[S * k + t] = x[j];
        }
    }
    __syncthreads();
    if constexpr (THREE) {
        for (int id = t; id < R0 * TB1; id += TPR) {
            const int o = id % TB1;
            u32* b = sm + S * (id / TB1) + o;
            u32 x[R1];
#pragma unroll
            for (int m = 0; m < R1; ++m) x[m] = b[TB1 * m];
            dif_regs<R1, true>(x, A.pk.rc.f, p, p2);
            const Tw* tw = A.tw + n + o;
#pragma unroll
            for (int j = 0; j < R1; ++j) {
                const int k = (int)rev_bits_c(j, PL.logr[1]);
                if (j > 0) {
                    const uint2 w = __ldg(reinterpret_cast<const uint2*>(tw + TB1 * k));
                    x[j] = mul_shoup(x[j], w.x, w.y, p);
                }
                b[TB1 * k] = x[j];
            }
        }
        __syncthreads();
    }
    if (!has) return;
    const u32 row = A.l1 ? col_slot_to_k1(s, A.colpl, A.l1) : s;
    u32* out = A.dst + (SLOT ? blockIdx.y * (size_t)A.job_stride : 0) + (size_t)row * n;
    for (int id = t; id < n / RL; id += TPR) {
        const u32* b = sm + S * (id % R0) + RL * (id / R0);
        u32 x[RL];
#pragma unroll
        for (int m = 0; m < RL; ++m) x[m] = b[m];
        dif_regs<RL>(x, A.pk.rc.f, p, p2);
#pragma unroll
        for (int j = 0; j < RL; ++j) out[id + (n / RL) * (int)rev_bits_c(j, PL.logr[PL.nlev - 1])] = red1(x[j], p);
    }
}

#endif  // __CUDACC__

}  // namespace cmb
