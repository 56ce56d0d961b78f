// Row passes of a bivariate product (2-D cyclic convolution) in the three
// passes of a long univariate one.
//
// A grid of 2^em rows (y) of 2^en words (x) is 2^l1 "column rows" of 2^(E+en)
// words, em = l1 + E: word y 2^en + x = y1 2^(E+en) + (y0 2^en + x) with
// y = y1 2^E + y0.  The product's column passes run the length-2^l1 transform
// over y1 as they do for a univariate product; what is left for the row
// passes of slot k1 is, over the 2^(E+en) words of its row, the radix-2^E
// transform over y0 with the twiddles w_m^(k1 y0) and a length-2^en transform
// of each of the 2^E rows over x -- no inter-pass twiddle along x.  Spectra
// stay in whatever order the passes leave them, F's and G's alike, so the
// product needs no transpose and no reordering: columns of F and G, G's rows
// (k_grid_fwd_g), F's rows with the pointwise product and the inverse rows
// (k_grid_mul_f), inverse columns.  With E, grids of up to 2^13 rows use the
// 2^10- and 2^11-row column kernels.
// Bound by integer issue like the univariate row kernels (k_row_fwd_g,
// k_row_mul_f), whose levels these are.  Measured on B200, 2^12 x 2^12, without
// copies: 249 us (with an event pair around each kernel: columns 77, G's rows
// 53, F's rows 101, inverse columns 39); row and column list transforms around
// two transposes took 543.
#pragma once
#include "large_product.cuh"

namespace cmb {

struct GridArgs {
    PrimeK pk;
    const Tw* __restrict__ twr;   // row plan tables of length 2^en: forward, inverse
    int twr_inv;
    const Tw* __restrict__ lead;  // E > 0: slot s's factors w_m^(k1 m) at 4 s + m (m < 2^E), then the inverse ones
                                  // times the scale, 4 2^l1 entries later
    int slots;                    // 2^l1
    Tw scale;                     // 2^32 / (grid words): undoes Montgomery's 2^-32 and the inverse's factor
    u32* wa;                      // F after the column pass; the row passes' output
    u32* wb;                      // G after the column pass; its spectrum
};

// Words of one CTA: a whole row, and at least 2^11.
__host__ __device__ constexpr int grid_log(int e, int l2) { return e + l2 > 11 ? e + l2 : 11; }
__host__ __device__ constexpr int grid_threads(int lt) { return 1 << (lt - 5); }
__host__ __device__ constexpr int grid_ctas(int lt) { return 1024 / grid_threads(lt); }

#ifdef __CUDACC__

// Forward levels LEV .. nlev-2 of every 2^L2-word row among 2^LT words.
template <int L2, int LEV, int LT, int T>
__device__ __forceinline__ void grid_fwd_levels(u32* sm, const GridArgs& A) {
    constexpr LevelPlan PL = row_plan(L2);
    if constexpr (LEV + 1 < PL.nlev) {
        using LV = SmallLevel<L2, LEV>;
        constexpr int R = LV::R, TB = LV::TB, B = LV::B;
        const u32 p = A.pk.p, p2 = A.pk.p2;
        for (int id = threadIdx.x; id < (1 << LT) / R; id += T) {
            const int o = id % TB, base = (id / TB) * B + o, bs = swz(base);
            u32 x[R];
#pragma unroll
            for (int m = 0; m < R; ++m) x[m] = sm[swz_task<TB, B>(base, bs, m)];
            dif_regs<R, true>(x, A.pk.rc.f, p, p2);
            Tw t[R];
            load_tw<R, TB>(t, A.twr + LV::TWOFF + o);
#pragma unroll
            for (int j = 1; j < R; ++j) x[j] = mul_shoup(x[j], t[j].w, t[j].wq, p);
#pragma unroll
            for (int m = 0; m < R; ++m) sm[swz_task<TB, B>(base, bs, m)] = x[m];
        }
        __syncthreads();
        grid_fwd_levels<L2, LEV + 1, LT, T>(sm, A);
    }
}

// Inverse levels LEV .. STOP.
template <int L2, int LEV, int STOP, int LT, int T>
__device__ __forceinline__ void grid_inv_levels(u32* sm, const GridArgs& A) {
    if constexpr (LEV >= STOP) {
        using LV = SmallLevel<L2, LEV>;
        constexpr int R = LV::R, TB = LV::TB, B = LV::B;
        const u32 p = A.pk.p, p2 = A.pk.p2;
        for (int id = threadIdx.x; id < (1 << LT) / R; id += T) {
            const int o = id % TB, base = (id / TB) * B + o, bs = swz(base);
            u32 x[R];
#pragma unroll
            for (int m = 0; m < R; ++m) x[m] = sm[swz_task<TB, B>(base, bs, m)];
            Tw t[R];
            load_tw<R, TB>(t, A.twr + A.twr_inv + LV::TWOFF + o);
#pragma unroll
            for (int j = 1; j < R; ++j) x[j] = mul_shoup(x[j], t[j].w, t[j].wq, p);
            dit_regs<R, true>(x, A.pk.rc.i, p, p2);
#pragma unroll
            for (int m = 0; m < R; ++m) sm[swz_task<TB, B>(base, bs, m)] = x[m];
        }
        __syncthreads();
        grid_inv_levels<L2, LEV - 1, STOP, LT, T>(sm, A);
    }
}

// The rows of this CTA in shared memory, through every forward level but the last.
template <int E, int L2, int LT, int T>
__device__ __forceinline__ void grid_forward(u32* sm, const u32* row, const GridArgs& A) {
    row_load_issue<LT, T>(sm, row);
    row_load_wait();
    __syncthreads();
    if constexpr (E > 0) {
        // over y0: words 2^L2 apart, times the slot's factors
        constexpr int R = 1 << E, TB = 1 << L2, B = TB << E;
        const u32 p = A.pk.p, p2 = A.pk.p2;
        for (int id = threadIdx.x; id < (1 << LT) / R; id += T) {
            const int o = id % TB, blk = id / TB, base = blk * B + o, bs = swz(base);
            const Tw* f = A.lead + 4 * ((size_t)blockIdx.x * ((1 << LT) / B) + blk);
            u32 x[R];
#pragma unroll
            for (int m = 0; m < R; ++m) {
                x[m] = sm[swz_task<TB, B>(base, bs, m)];
                if (m > 0) {
                    const uint2 w = __ldg(reinterpret_cast<const uint2*>(f + m));
                    x[m] = mul_shoup(x[m], w.x, w.y, p);
                }
            }
            dif_regs<R>(x, A.pk.rc.f, p, p2);
#pragma unroll
            for (int m = 0; m < R; ++m) sm[swz_task<TB, B>(base, bs, m)] = x[m];
        }
        __syncthreads();
    }
    grid_fwd_levels<L2, 0, LT, T>(sm, A);
}

// G's rows: the spectrum over G, its 32-word groups quad-interleaved as k_row_fwd_g leaves them.
template <int E, int L2>
__global__ void __launch_bounds__(grid_threads(grid_log(E, L2)), grid_ctas(grid_log(E, L2)))
    k_grid_fwd_g(const __grid_constant__ GridArgs A) {
    constexpr int LT = grid_log(E, L2), T = grid_threads(LT), N = 1 << LT;
    extern __shared__ __align__(16) u32 sm[];
    u32* row = A.wb + (size_t)blockIdx.x * N;
    pdl_wait();  // the column pass
    pdl_trigger();  // after it: k_grid_mul_f reads F's columns before its own wait
    grid_forward<E, L2, LT, T>(sm, row, A);
    for (int r = threadIdx.x; r < N / 32; r += T) {
        u32 x[32];
        load_row32(x, sm, r * 32);
        dif_regs<32>(x, A.pk.rc.f, A.pk.p, A.pk.p2);
#pragma unroll
        for (int c = 0; c < 8; ++c)
            *reinterpret_cast<uint4*>(row + c * (N / 8) + 4 * r) =
                make_uint4(x[4 * c], x[4 * c + 1], x[4 * c + 2], x[4 * c + 3]);
    }
}

// F's rows, the pointwise product with G's spectrum, the inverse rows over F.
template <int E, int L2>
__global__ void __launch_bounds__(grid_threads(grid_log(E, L2)), grid_ctas(grid_log(E, L2)))
    k_grid_mul_f(const __grid_constant__ GridArgs A) {
    constexpr int LT = grid_log(E, L2), T = grid_threads(LT), N = 1 << LT;
    constexpr LevelPlan PL = row_plan(L2);
    extern __shared__ __align__(16) u32 sm[];
    const u32 p = A.pk.p, p2 = A.pk.p2, pinv = A.pk.pinv_neg;
    u32* row = A.wa + (size_t)blockIdx.x * N;
    const u32* rowG = A.wb + (size_t)blockIdx.x * N;
    pdl_trigger();
    // F's forward rows depend only on the column passes, which G's row kernel
    // waits for before it allows this launch; G's spectrum is read after pdl_wait
    grid_forward<E, L2, LT, T>(sm, row, A);
    pdl_wait();
    for (int r = threadIdx.x; r < N / 32; r += T) {
        u32 x[32];
        load_row32(x, sm, r * 32);
        dif_regs<32>(x, A.pk.rc.f, p, p2);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const uint4 g = __ldg(reinterpret_cast<const uint4*>(rowG + c * (N / 8) + 4 * r));
            x[4 * c] = mul_mont(x[4 * c], g.x, p, pinv);
            x[4 * c + 1] = mul_mont(x[4 * c + 1], g.y, p, pinv);
            x[4 * c + 2] = mul_mont(x[4 * c + 2], g.z, p, pinv);
            x[4 * c + 3] = mul_mont(x[4 * c + 3], g.w, p, pinv);
        }
        dit_regs<32>(x, A.pk.rc.i, p, p2);
        store_row32(sm, r * 32, x);
    }
    __syncthreads();
    grid_inv_levels<L2, PL.nlev - 2, (E > 0 ? 0 : 1), LT, T>(sm, A);
    if constexpr (E > 0) {
        constexpr int R = 1 << E, TB = 1 << L2, B = TB << E;
        for (int id = threadIdx.x; id < N / R; id += T) {
            const int o = id % TB, blk = id / TB, base = blk * B + o, bs = swz(base);
            const Tw* f = A.lead + 4 * (A.slots + (size_t)blockIdx.x * (N / B) + blk);
            u32 x[R];
#pragma unroll
            for (int m = 0; m < R; ++m) x[m] = sm[swz_task<TB, B>(base, bs, m)];
            dit_regs<R>(x, A.pk.rc.i, p, p2);
#pragma unroll
            for (int m = 0; m < R; ++m) {
                const uint2 w = __ldg(reinterpret_cast<const uint2*>(f + m));
                row[base + TB * m] = mul_shoup(x[m], w.x, w.y, p);
            }
        }
    } else {
        using LV = SmallLevel<L2, 0>;
        constexpr int R = LV::R, TB = LV::TB, B = LV::B;
        for (int id = threadIdx.x; id < N / R; id += T) {
            const int o = id % TB, base = (id / TB) * B + o, bs = swz(base);
            u32 x[R];
            Tw t[R];
            load_tw<R, TB>(t, A.twr + A.twr_inv + o);
#pragma unroll
            for (int m = 0; m < R; ++m) {
                x[m] = sm[swz_task<TB, B>(base, bs, m)];
                if (m > 0) x[m] = mul_shoup(x[m], t[m].w, t[m].wq, p);
            }
            dit_regs<R, true>(x, A.pk.rc.i, p, p2);
#pragma unroll
            for (int m = 0; m < R; ++m) row[base + TB * m] = mul_shoup(x[m], A.scale.w, A.scale.wq, p);
        }
    }
}

#endif  // __CUDACC__

}  // namespace cmb
