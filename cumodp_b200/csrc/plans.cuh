// Compile-time level plans for the shared-memory transforms.
#pragma once
#include "ntt_engine.cuh"

namespace cmb {

// Plan for a contiguous transform of length 2^logl held in shared memory.
// The last level always has radix 32: every earlier level then has at least
// 32 tasks per block, so 32 lanes touch 32 consecutive words (no bank
// conflicts), and the last level reads whole 32-word rows with 16-byte
// accesses through the swizzle.  From 2^12 on three levels: a fourth costs a
// Shoup product, a twiddle and a shared-memory exchange per word (2^14-word
// rows, g + f of a 2^24 product: 56 + 113 us with {3, 3, 3, 5}, 58 + 103 with
// {4, 5, 5}).
__host__ __device__ constexpr LevelPlan row_plan(int logl) {
    switch (logl) {
        case 5: return LevelPlan{1, {5}};
        case 6: return LevelPlan{2, {1, 5}};
        case 7: return LevelPlan{2, {2, 5}};
        case 8: return LevelPlan{2, {3, 5}};
        case 9: return LevelPlan{2, {4, 5}};
        case 10: return LevelPlan{3, {2, 3, 5}};
        case 11: return LevelPlan{3, {3, 3, 5}};
        case 12: return LevelPlan{3, {3, 4, 5}};
        case 13: return LevelPlan{3, {4, 4, 5}};
        case 14: return LevelPlan{3, {4, 5, 5}};
        default: return LevelPlan{0, {0}};
    }
}

// Plan for a batch of interleaved columns (lane = column): bank conflicts do
// not depend on the radix, so fewer, wider levels are used (two levels up to
// 2^10 rows: every element goes through shared memory twice).
__host__ __device__ constexpr LevelPlan col_plan(int logl) {
    switch (logl) {
        case 1: return LevelPlan{1, {1}};
        case 2: return LevelPlan{1, {2}};
        case 3: return LevelPlan{1, {3}};
        case 4: return LevelPlan{1, {4}};
        case 5: return LevelPlan{2, {2, 3}};
        case 6: return LevelPlan{2, {3, 3}};
        case 7: return LevelPlan{2, {3, 4}};
        case 8: return LevelPlan{2, {4, 4}};
        case 9: return LevelPlan{2, {4, 5}};
        case 10: return LevelPlan{2, {5, 5}};
        case 11: return LevelPlan{3, {3, 4, 4}};
        case 12: return LevelPlan{3, {4, 4, 4}};
        default: return LevelPlan{0, {0}};
    }
}

// Twiddle entries (one direction) of the column plan of length 2^logl.
__host__ __device__ constexpr int col_tw_entries(int logl) {
    int n = 0, lb = logl;
    const LevelPlan pl = col_plan(logl);
    for (int i = 0; i + 1 < pl.nlev; ++i) { n += 1 << lb; lb -= pl.logr[i]; }
    return n;
}
// Column tiles in shared memory (k_col_fwd, k_col_inv: 2^11-row columns;
// shorter ones are col_direct.cuh's): 16 adjacent columns x 2^logl rows on 16
// warps, one CTA per SM.  A warp has two tasks, one per half-warp, and a
// 16-word pad after every 2^col_pad_log rows (the plan's last radix) makes the
// two half-warps read opposite halves of the banks.
constexpr int kColTileCols = 16, kColTileWarps = 16;
__host__ __device__ constexpr int col_pad_log(int logl) { return col_plan(logl).logr[col_plan(logl).nlev - 1]; }
__host__ __device__ constexpr int col_tile_words(int logl) {
    return ((1 << logl) + ((1 << logl) >> col_pad_log(logl))) * kColTileCols;
}
// Dynamic shared memory of a column CTA: the tile and its twiddles.
__host__ __device__ constexpr int col_smem_bytes(int logl) { return col_tile_words(logl) * 4 + col_tw_entries(logl) * 8; }

// A single product (no batch) of transform length 2^logn uses the three-pass
// kernels from this length on, even where one CTA could hold it: spread over
// many CTAs it finishes sooner than on one SM.
__host__ __device__ constexpr int single_large_min_log() { return 13; }

// Threads of the three-pass row kernel: 2^14-word rows use 1024 threads with
// at most 64 registers each (32 warps per SM; the plan's twiddled levels
// have radix <= 8 so both operands fit), shorter rows the single-CTA count.
__host__ __device__ constexpr int row_threads(int logl);

// Threads and products per CTA for the fused single-CTA product of length L.
__host__ __device__ constexpr int small_threads(int logl) { return logl >= 12 ? (1 << (logl - 5)) : 128; }
__host__ __device__ constexpr int small_ppc(int logl) { return logl >= 12 ? 1 : (1 << (12 - logl)); }
// Resident CTAs per SM the fused single-CTA product is compiled for: six
// 32 KiB CTAs of 128 threads (80 registers) for lengths <= 2^12, three
// 64 KiB CTAs for 2^13, one 128 KiB CTA for 2^14.
__host__ __device__ constexpr int small_ctas(int logl) { return logl <= 12 ? 6 : logl == 13 ? 3 : 1; }
__host__ __device__ constexpr int row_threads(int logl) { return logl == 14 ? 1024 : small_threads(logl); }
// Threads of the split row kernels (one operand row per CTA): one per
// 32-word row of the last level.
__host__ __device__ constexpr int rowsplit_threads(int logl) { return logl >= 10 ? (1 << (logl - 5)) : 32; }
// Resident CTAs per SM the split row kernels are compiled for: 1024 threads
// of 64 registers.
__host__ __device__ constexpr int rowsplit_ctas(int logl) { return (1024 / rowsplit_threads(logl) < 32 ? 1024 / rowsplit_threads(logl) : 32); }

}  // namespace cmb
