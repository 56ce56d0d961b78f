// One product in one launch, for latency: transforms of n = 2^5 .. 2^16 words.
//
// A single product is bound by its serial chain -- launches, global loads,
// barriers, the instructions of one thread's tasks -- and not by any rate, so
// these kernels give every thread one radix-4..16 task per level (the
// throughput kernels of small_product.cuh give it radix 32 and up to eight
// products per CTA) and keep the whole product in shared memory:
//   n <= 2^11  one CTA, 2n/8 threads;
//   n >= 2^12  a cluster of 16 CTAs.  The first level has radix 16 and its
//              block j is an independent transform of n/16 words, so each
//              CTA runs 1/16 of that level's tasks straight from global
//              memory, sends output j to CTA j over distributed shared
//              memory, transforms its own block of both operands, multiplies,
//              transforms back, and sends the words home for the last
//              inverse level, which stores the result: two exchanges in all.
// Twiddles of the levels inside a CTA are copied to shared memory while the
// operands are on their way; those of the leading level are read from global
// memory, one coalesced word pair per output.
// Measured on B200 (device time of one product, 20 calls in a graph; before:
// k_small_product on one CTA up to 2^12, the four kernels of the three-pass
// product from 2^13 on):
//   2^5    8.0 ->  1.5 us     2^9   11.7 ->  2.5 us     2^13  12.0 ->  4.5 us
//   2^7    9.5 ->  2.2 us     2^11  13.5 ->  4.0 us     2^14  12.3 ->  5.2 us
//   2^8   10.1 ->  2.4 us     2^12  16.9 ->  4.4 us     2^16  14.8 -> 11.5 us
// At 2^17 a block of both operands, the words on their way home and the
// twiddles no longer fit one CTA's shared memory; the three-pass kernels
// (17.4 us there) run from that length on.
#pragma once
#include "small_product.cuh"

namespace cmb {

constexpr int kClusterCtas = 16;
constexpr int kLeadLog = 4;  // log2 of the leading level's radix: one block per CTA of the cluster

// Levels of a block of 2^logl words held by one CTA.  The last level's radix
// is 8: one thread runs it on both operands, multiplies and starts the
// inverse in registers.
__host__ __device__ constexpr LevelPlan lat_plan(int logl) {
    switch (logl) {
        case 5: return LevelPlan{2, {2, 3}};
        case 6: return LevelPlan{2, {3, 3}};
        case 7: return LevelPlan{3, {2, 2, 3}};
        case 8: return LevelPlan{3, {3, 2, 3}};
        case 9: return LevelPlan{3, {3, 3, 3}};
        case 10: return LevelPlan{3, {4, 3, 3}};
        case 11: return LevelPlan{3, {4, 4, 3}};
        case 12: return LevelPlan{4, {3, 3, 3, 3}};
        default: return LevelPlan{0, {0}};
    }
}
// Entries (one direction) of the block's twiddle table: level i's entry
// (task o, slot j) at off_i + j TB_i + o, so that a warp's tasks read
// consecutive entries.
__host__ __device__ constexpr int lat_entries(int logl) {
    int n = 0, lb = logl;
    const LevelPlan pl = lat_plan(logl);
    for (int i = 0; i + 1 < pl.nlev; ++i) { n += 1 << lb; lb -= pl.logr[i]; }
    return n;
}
// One thread per radix-8 task of the two operands, at most 512 (1024 threads for
// 2^12-word blocks: 11.7 us against 11.5 at 2^16).
__host__ __device__ constexpr int lat_threads(int logl) {
    return logl <= 7 ? 32 : logl >= 11 ? 512 : (1 << (logl - 2));
}
// Word index in shared memory: 32 consecutive words, words 8 apart (the last
// level) and 64-word blocks read 8 words at a time all spread over the banks.
__host__ __device__ constexpr int lat_pad(int i) { return i + (i >> 5) + ((i >> 6) << 3); }
__host__ __device__ constexpr int lat_words(int logl) { return lat_pad((1 << logl) - 1) + 1; }
// Shared memory: both operands' blocks, in a cluster the words on their way
// home, and the block's twiddles of both directions.
__host__ __device__ constexpr size_t lat_smem(int logl, int cluster) {
    const size_t words = (size_t)2 * ((lat_words(logl) + 3) & ~3) + (cluster > 1 ? (size_t)1 << logl : 0);
    return words * sizeof(u32) + (size_t)2 * lat_entries(logl) * sizeof(Tw);
}

// Exponent e of entry t of latency_tables' array: the entry is w^e for the
// product's primitive 2^logn-th root w.  The block's levels (2^logl words),
// forward then inverse, and for logl < logn the leading level, forward then
// inverse (an inverse entry's exponent is 2^logn less the forward one's).
struct LatExponent {
    LevelPlan pl;
    int logl, logn, block;  // block: lat_entries(logl)
    __host__ __device__ u32 operator()(u32 t) const {
        const u32 n = 1u << logn;
        u32 e, q = t < 2u * block ? t % block : (t - 2u * block) % n;
        const bool inv = t < 2u * block ? t >= (u32)block : t - 2u * block >= n;
        if (t < 2u * block) {
            int i = 0, lb = logl;
            while (q >= 1u << lb) {
                q -= 1u << lb;
                lb -= pl.logr[i++];
            }
            const int lt = lb - pl.logr[i];  // 2^lt tasks a block
            e = ((q & ((1u << lt) - 1)) * rev_bits(q >> lt, pl.logr[i])) << (logn - lb);
        } else {
            e = (q & ((1u << logl) - 1)) * rev_bits(q >> logl, logn - logl);
        }
        return inv ? (n - e) & (n - 1) : e;
    }
};

struct LatPrime {
    PrimeK pk;
    Tw scale;        // 2^32 / n (undoes Montgomery's 2^-32 and the inverse's n)
    Tw r32;          // 2^32 mod p
    const Tw* tw;    // block tables: forward, then inverse
    const Tw* lead;  // leading level: entry (o, j) at j n/16 + o; forward, then inverse
};
// NP products of the same lengths, one per prime (grid dimension y): prime r's
// operands at a + r astride, b + r bstride (elements), its residues at h + r
// hstride.
template <int NP>
struct LatArgs {
    LatPrime pr[NP];
    const void *a, *b;
    u32* h;
    int la, lb, lh;
    long long astride, bstride, hstride;
};

#ifdef __CUDACC__

template <int LOGL, int LEV>
struct LatLevel {
    static constexpr LevelPlan PL = lat_plan(LOGL);
    static constexpr int R = 1 << PL.logr[LEV];
    static constexpr int LOGB = [] {
        int lb = LOGL;
        for (int i = 0; i < LEV; ++i) lb -= PL.logr[i];
        return lb;
    }();
    static constexpr int B = 1 << LOGB, TB = B / R;
    static constexpr int TWOFF = [] {
        int n = 0, lb = LOGL;
        for (int i = 0; i < LEV; ++i) { n += 1 << lb; lb -= PL.logr[i]; }
        return n;
    }();
};

__device__ __forceinline__ u32 cluster_map(const void* smem, u32 rank) {
    u32 a = (u32)__cvta_generic_to_shared(smem), r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_store(u32 addr, u32 v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Forward levels LEV .. nlev-2 of both operands' blocks, one operand per task.
template <int LOGL, int LEV, int T>
__device__ __forceinline__ void lat_fwd_levels(u32* sm, const Tw* tws, const PrimeK& pk) {
    using LV = LatLevel<LOGL, LEV>;
    constexpr int L = 1 << LOGL, R = LV::R, TB = LV::TB, B = LV::B, W = (lat_words(LOGL) + 3) & ~3;
    if constexpr (LEV + 1 < LV::PL.nlev) {
        const u32 p = pk.p, p2 = pk.p2;
        for (int id = threadIdx.x; id < 2 * (L / R); id += T) {
            const int rest = id % (L / R), o = rest % TB, base = (rest / TB) * B + o;
            u32* s = sm + (id / (L / R)) * W;
            u32 x[R];
#pragma unroll
            for (int m = 0; m < R; ++m) x[m] = s[lat_pad(base + TB * m)];
            dif_regs<R, true>(x, pk.rc.f, p, p2);
#pragma unroll
            for (int j = 1; j < R; ++j) {
                const Tw t = tws[LV::TWOFF + j * TB + o];
                x[j] = mul_shoup(x[j], t.w, t.wq, p);
            }
#pragma unroll
            for (int m = 0; m < R; ++m) s[lat_pad(base + TB * m)] = x[m];
        }
        __syncthreads();
        lat_fwd_levels<LOGL, LEV + 1, T>(sm, tws, pk);
    }
}

// Inverse levels LEV .. 0 of the product's block; the last one hands element
// i of the block to put(i, value in [0, 4p)).
template <int LOGL, int LEV, int T, class Put>
__device__ __forceinline__ void lat_inv_levels(u32* sm, const Tw* twi, const PrimeK& pk, Put put) {
    if constexpr (LEV >= 0) {
        using LV = LatLevel<LOGL, LEV>;
        constexpr int L = 1 << LOGL, R = LV::R, TB = LV::TB, B = LV::B;
        const u32 p = pk.p, p2 = pk.p2;
        for (int id = threadIdx.x; id < L / R; id += T) {
            const int o = id % TB, base = (id / TB) * B + o;
            u32 x[R];
#pragma unroll
            for (int m = 0; m < R; ++m) x[m] = sm[lat_pad(base + TB * m)];
#pragma unroll
            for (int j = 1; j < R; ++j) {
                const Tw t = twi[LV::TWOFF + j * TB + o];
                x[j] = mul_shoup(x[j], t.w, t.wq, p);
            }
            dit_regs<R, true>(x, pk.rc.i, p, p2);
#pragma unroll
            for (int m = 0; m < R; ++m) {
                if constexpr (LEV > 0) sm[lat_pad(base + TB * m)] = x[m];
                else put(base + TB * m, x[m]);
            }
        }
        if constexpr (LEV > 0) __syncthreads();
        lat_inv_levels<LOGL, LEV - 1, T>(sm, twi, pk, put);
    }
}

// Word i of an operand in [0, 2p), zero past its end: a 32-bit word, or the
// residue of a signed 64-bit one (its two halves' residues, one Shoup
// product each, negated for a negative number).
template <bool WIDE>
struct LatWord;
template <>
struct LatWord<false> {
    typedef u32 T;
    static __device__ __forceinline__ u32 reduce(u32 v, const LatPrime& P) {
        return mul_shoup(v, 1u, P.pk.one_q, P.pk.p);
    }
};
template <>
struct LatWord<true> {
    typedef long long T;
    static __device__ __forceinline__ u32 reduce(long long v, const LatPrime& P) {
        const u32 p = P.pk.p, p2 = P.pk.p2;
        const u64 m = v < 0 ? 0ull - (u64)v : (u64)v;
        const u32 r = red2(mul_shoup((u32)m, 1u, P.pk.one_q, p) + mul_shoup((u32)(m >> 32), P.r32.w, P.r32.wq, p), p2);
        return v < 0 ? red2(p2 - r, p2) : r;  // p2 - 0 is p2, which red2 takes to 0
    }
};

// One product per prime: blocks of 2^LOGL words, CL = 1 (n = 2^LOGL) or a
// cluster of 16 CTAs (n = 2^(LOGL + 4)); WIDE: signed 64-bit operands.
template <int LOGL, int CL, int NP, bool WIDE>
__global__ void __launch_bounds__(lat_threads(LOGL), 1) k_latency_product(const __grid_constant__ LatArgs<NP> A) {
    constexpr int L = 1 << LOGL, T = lat_threads(LOGL), W = (lat_words(LOGL) + 3) & ~3;
    constexpr LevelPlan PL = lat_plan(LOGL);
    constexpr int NE = lat_entries(LOGL);
    constexpr int CH = L / kClusterCtas;  // leading-level tasks of one CTA
    static_assert(CL == 1 || CL == kClusterCtas, "one CTA, or one CTA per leading block");
    static_assert(PL.nlev >= 2 && PL.logr[PL.nlev - 1] == 3, "the last level runs in one thread per 8 words");
    static_assert(NE % 2 == 0, "16-byte copies");
    extern __shared__ __align__(16) u32 sm[];  // F's block, G's block, [words on their way home], twiddles
    u32* home = sm + 2 * W;
    Tw* tws = reinterpret_cast<Tw*>(home + (CL > 1 ? L : 0));
    using Word = LatWord<WIDE>;
    typedef typename Word::T In;
    const int prime = NP > 1 ? (int)blockIdx.y : 0;
    const LatPrime& P = A.pr[prime];
    const In* const opa = (const In*)A.a + (NP > 1 ? prime * A.astride : 0);
    const In* const opb = (const In*)A.b + (NP > 1 ? prime * A.bstride : 0);
    u32* const h = A.h + (NP > 1 ? prime * A.hstride : 0);
    const u32 p = P.pk.p, p2 = P.pk.p2;
    if constexpr (NP > 1) pdl_trigger();
    const u32 rank = CL > 1 ? blockIdx.x : 0;
    if constexpr (CL > 1) cluster_arrive();  // waited for before the first remote store
    for (int i = threadIdx.x; i < NE; i += T) {
        const unsigned d = (unsigned)__cvta_generic_to_shared(tws + 2 * i);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(P.tw + 2 * i) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");

    if constexpr (CL == 1) {
        // both operands, reduced to [0, 2p), zero past their ends
        In v[2 * L / T];
#pragma unroll
        for (int u = 0; u < 2 * L / T; ++u) {
            const int idx = threadIdx.x + u * T, i = idx % L;
            const bool second = idx >= L;
            v[u] = i < (second ? A.lb : A.la) ? __ldg((second ? opb : opa) + i) : In(0);
        }
#pragma unroll
        for (int u = 0; u < 2 * L / T; ++u) {
            const int idx = threadIdx.x + u * T;
            sm[(idx / L) * W + lat_pad(idx % L)] = Word::reduce(v[u], P);
        }
    } else {
        // leading level, radix 16: task o reads words o + L m, its output j
        // is word o of block j
        static_assert(2 * CH <= T && 2 * CH % 32 == 0, "one task per thread, whole warps");
        const bool has = threadIdx.x < 2 * CH;
        const int op = threadIdx.x / CH, o = (int)rank * CH + threadIdx.x % CH;
        u32 x[16];
        if (has) {
            const In* src = op ? opb : opa;
            const int len = op ? A.lb : A.la;
            Tw t[16];
            In v[16];
#pragma unroll
            for (int m = 0; m < 16; ++m) v[m] = o + L * m < len ? __ldg(src + o + L * m) : In(0);
#pragma unroll
            for (int j = 1; j < 16; ++j) {
                const uint2 w = __ldg(reinterpret_cast<const uint2*>(P.lead + j * L + o));
                t[j] = Tw{w.x, w.y};
            }
#pragma unroll
            for (int m = 0; m < 16; ++m) x[m] = Word::reduce(v[m], P);
            dif_regs<16, true>(x, P.pk.rc.f, p, p2);
#pragma unroll
            for (int j = 1; j < 16; ++j) x[j] = mul_shoup(x[j], t[j].w, t[j].wq, p);
        }
        cluster_wait();  // every CTA of the cluster has started
        if (has) {
            u32* dst = sm + op * W + lat_pad(o);
#pragma unroll
            for (int j = 0; j < 16; ++j) cluster_store(cluster_map(dst, j), x[j]);
        }
        cluster_arrive();
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    if constexpr (CL > 1) cluster_wait();  // this CTA's blocks are complete
    lat_fwd_levels<LOGL, 0, T>(sm, tws, P.pk);

    // last forward level of both operands, pointwise product, first inverse level
    for (int id = threadIdx.x; id < L / 8; id += T) {
        u32 f[8], g[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            f[m] = sm[lat_pad(8 * id + m)];
            g[m] = sm[W + lat_pad(8 * id + m)];
        }
        dif_regs<8>(f, P.pk.rc.f, p, p2);
        dif_regs<8>(g, P.pk.rc.f, p, p2);
#pragma unroll
        for (int m = 0; m < 8; ++m)
            f[m] = mul_shoup(mul_mont(f[m], g[m], p, P.pk.pinv_neg), P.scale.w, P.scale.wq, p);
        dit_regs<8>(f, P.pk.rc.i, p, p2);
#pragma unroll
        for (int m = 0; m < 8; ++m) sm[lat_pad(8 * id + m)] = f[m];
    }
    __syncthreads();

    if constexpr (CL == 1) {
        lat_inv_levels<LOGL, PL.nlev - 2, T>(sm, tws + NE, P.pk, [&](int i, u32 v) {
            if (i < A.lh) h[i] = red1(red2(v, p2), p);
        });
    } else {
        lat_inv_levels<LOGL, PL.nlev - 2, T>(sm, tws + NE, P.pk, [&](int i, u32 v) {
            cluster_store(cluster_map(home + rank * CH + i % CH, i / CH), v);
        });
        cluster_arrive();
        // last inverse level: task o takes word o of every block
        const int o = (int)(rank * CH + threadIdx.x);
        Tw t[16];
        if (threadIdx.x < CH) {
#pragma unroll
            for (int j = 1; j < 16; ++j) {
                const uint2 w = __ldg(reinterpret_cast<const uint2*>(P.lead + (16 + j) * L + o));
                t[j] = Tw{w.x, w.y};
            }
        }
        cluster_wait();
        if (threadIdx.x < CH) {
            u32 x[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) x[j] = home[j * CH + threadIdx.x];
#pragma unroll
            for (int j = 1; j < 16; ++j) x[j] = mul_shoup(x[j], t[j].w, t[j].wq, p);
            dit_regs<16, true>(x, P.pk.rc.i, p, p2);
#pragma unroll
            for (int m = 0; m < 16; ++m)
                if (o + L * m < A.lh) h[o + L * m] = red1(red2(x[m], p2), p);
        }
    }
}

// One level of a subproduct tree (cumodp_subproduct_level_dev) for transforms
// of 2^LOGL = n >= 2l words: pair j's monic polynomials x^l + a and x^l + b
// (l words each, consecutive) go in with their leading coefficient, and their
// product mod x^n - 1 has the 2l words wanted, except that for n = 2l the
// leading x^(2l) wraps onto the constant term.  So the x^l (a + b) term costs
// nothing, and no job table is made or uploaded: a job is its index.
// Persistent CTAs (the twiddles are copied once); the next pair's words are
// loaded while the current pair is transformed.  One operand per task and
// radix 8 last keep a thread's data in 16 registers: the batch kernel's
// radix-32 level holds 64 and spends as long on it as on the rest.  Bound by
// integer issue (68 % of the issue slots).  Measured on B200, with the batch
// kernel, its job upload and the fix-up pass before: 2048 pairs of degree 512
// 41 -> 23 us, 32768 of them 583 -> 263 us, 65536 pairs of degree 16 1102 -> 39
// us (a job table a call).
struct LevelArgs {
    LatPrime pr;
    const u32* in;
    u32* out;
    int l, npairs;
};
__host__ __device__ constexpr int level_threads(int logl) { return logl <= 8 ? 32 : 1 << (logl - 3); }
__host__ __device__ constexpr int level_ctas(int logl) { return logl <= 8 ? 24 : logl <= 10 ? 1024 / level_threads(logl) : logl == 11 ? 4 : 2; }

template <int LOGL>
__global__ void __launch_bounds__(level_threads(LOGL), level_ctas(LOGL)) k_monic_level(const __grid_constant__ LevelArgs A) {
    constexpr int L = 1 << LOGL, T = level_threads(LOGL), W = (lat_words(LOGL) + 3) & ~3;
    constexpr LevelPlan PL = lat_plan(LOGL);
    constexpr int NE = lat_entries(LOGL), NV = 2 * L / T;
    extern __shared__ __align__(16) u32 sm[];  // F, G, twiddles
    Tw* tws = reinterpret_cast<Tw*>(sm + 2 * W);
    const LatPrime& P = A.pr;
    const u32 p = P.pk.p, p2 = P.pk.p2;
    for (int i = threadIdx.x; i < NE; i += T) {
        const unsigned d = (unsigned)__cvta_generic_to_shared(tws + 2 * i);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(P.tw + 2 * i) : "memory");
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    u32 v[NV];
    auto load = [&](u32 j) {
        const u32* src = A.in + (size_t)2 * j * A.l;
#pragma unroll
        for (int u = 0; u < NV; ++u) {
            const int idx = threadIdx.x + u * T, i = idx % L, at = (idx >= L ? A.l : 0) + i;
            v[u] = i < A.l ? __ldg(src + at) : i == A.l ? 1u : 0u;
        }
    };
    u32 j = blockIdx.x;
    const u32 npairs = A.npairs;
    if (j < npairs) load(j);
    for (; j < npairs; j += gridDim.x) {
#pragma unroll
        for (int u = 0; u < NV; ++u) {
            const int idx = threadIdx.x + u * T;
            sm[(idx / L) * W + lat_pad(idx % L)] = mul_shoup(v[u], 1u, P.pk.one_q, p);
        }
        __syncthreads();
        if (j + gridDim.x < npairs) load(j + gridDim.x);
        lat_fwd_levels<LOGL, 0, T>(sm, tws, P.pk);
        for (int id = threadIdx.x; id < L / 8; id += T) {
            u32 f[8], g[8];
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                f[m] = sm[lat_pad(8 * id + m)];
                g[m] = sm[W + lat_pad(8 * id + m)];
            }
            dif_regs<8>(f, P.pk.rc.f, p, p2);
            dif_regs<8>(g, P.pk.rc.f, p, p2);
#pragma unroll
            for (int m = 0; m < 8; ++m)
                f[m] = mul_shoup(mul_mont(f[m], g[m], p, P.pk.pinv_neg), P.scale.w, P.scale.wq, p);
            dit_regs<8>(f, P.pk.rc.i, p, p2);
#pragma unroll
            for (int m = 0; m < 8; ++m) sm[lat_pad(8 * id + m)] = f[m];
        }
        __syncthreads();
        u32* out = A.out + (size_t)2 * j * A.l;
        lat_inv_levels<LOGL, PL.nlev - 2, T>(sm, tws + NE, P.pk, [&](int i, u32 x) {
            if (i < 2 * A.l) {
                u32 c = red1(red2(x, p2), p);
                if (i == 0 && 2 * A.l == L) c = c ? c - 1 : p - 1;
                out[i] = c;
            }
        });
        __syncthreads();  // the last inverse level has read its words
    }
}

#endif  // __CUDACC__

}  // namespace cmb
