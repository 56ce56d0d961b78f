// Host-side check of every shared-memory and table index map the kernels use,
// for every plan the library instantiates.  The maps are the kernels' own
// __host__ __device__ functions (compiled here for the host), so an
// out-of-bounds or colliding index shows up here instead of on a GPU.
//
//   rows:    every non-last level of every row plan (lengths 2^5..2^14,
//            products of one and of several operand pairs per CTA) touches
//            each word of its buffer exactly once, swz_task equals the plain
//            swizzle, the last level's 16-byte quads tile the buffer, and the
//            twiddle reads cover the level's entries of the plan's table;
//   staged columns (2^11 rows): tile_row is injective and in bounds, tile_step
//            equals tile_row differences for every level task, and the two
//            half-warps read opposite halves of the banks;
//   register columns (2^1..2^10 rows): the exchange between the two levels is a
//            bijection within shared memory, rows are read and written once;
//   natural-order rows (2^6..2^14 words): every level touches each word once,
//            outputs are a permutation, shared memory and tables are in bounds;
//   bivariate rows: the same for the leading level and the levels over x;
//   orders:  col_slot_to_k1 is bit reversal for every column plan;
//   row factor tables (rows of 2^11..2^14 words): every level-0 task reads
//            its two entries inside the table, the two digits recompose the
//            task index, and the row kernels' shared memory fits the SM;
//   one-launch products and subproduct levels: padded addresses in bounds and
//            distinct, level tasks cover each block once, twiddle reads in
//            bounds, shared memory fits; the table builders' exponents;
//   Shoup quotients from the double estimate equal floor(w 2^32 / p);
//   the quad-interleaved row spectrum is a permutation with warp-contiguous runs.
#include <cstdio>
#include <set>
#include <vector>

#include "../cumodp_b200/csrc/col_direct.cuh"
#include "../cumodp_b200/csrc/grid_product.cuh"
#include "../cumodp_b200/csrc/large_product.cuh"
#include "../cumodp_b200/csrc/latency_product.cuh"
#include "../cumodp_b200/csrc/row_natural.cuh"

using namespace cmb;

static int failures = 0;
#define CHECK(c, ...)                          \
    do {                                       \
        if (!(c)) {                            \
            if (failures < 20) {               \
                std::printf("FAIL: " __VA_ARGS__); \
                std::printf("\n");             \
            }                                  \
            ++failures;                        \
        }                                      \
    } while (0)

template <int LOGL, int LEV>
void row_level(int ppc) {
    using LV = SmallLevel<LOGL, LEV>;
    constexpr int L = 1 << LOGL, R = LV::R, TB = LV::TB, B = LV::B;
    std::vector<int> seen((size_t)ppc * 2 * L, 0), read((size_t)plan_tw_entries(row_plan(LOGL), LOGL), 0);
    for (int q = 0; q < ppc; ++q)
        for (int op = 0; op < 2; ++op)
            for (int rest = 0; rest < L / R; ++rest) {
                const int blk = rest / TB, o = rest % TB;
                const int base = q * 2 * L + op * L + blk * B + o;
                const int bs = swz(base);
                for (int m = 0; m < R; ++m) {
                    const int a = swz_task<TB, B>(base, bs, m);
                    CHECK((a == swz(base + TB * m)), "row L=%d lev=%d swz_task", LOGL, LEV);
                    CHECK(a >= 0 && a < (int)seen.size(), "row L=%d lev=%d out of range", LOGL, LEV);
                    if (a >= 0 && a < (int)seen.size()) seen[a]++;
                }
                // twiddles of this task: slot j at j TB + o (load_tw)
                for (int j = 0; j < R; ++j) {
                    const size_t t = (size_t)(LV::TWOFF + j * TB + o);
                    CHECK(t < read.size(), "row L=%d lev=%d twiddle index", LOGL, LEV);
                    if (t < read.size()) read[t]++;
                }
            }
    for (size_t i = 0; i < seen.size(); ++i) CHECK(seen[i] == 1, "row L=%d lev=%d word %zu hit %d", LOGL, LEV, i, seen[i]);
    // every task of the level reads its own entries, once per block and operand
    for (size_t t = 0; t < read.size(); ++t)
        CHECK(read[t] == ((int)t >= LV::TWOFF && (int)t < LV::TWOFF + B ? ppc * 2 * (L / B) : 0),
              "row L=%d lev=%d twiddle %zu read %d times", LOGL, LEV, t, read[t]);
}

template <int LOGL, int LEV>
void row_levels(int ppc) {
    constexpr LevelPlan PL = row_plan(LOGL);
    if constexpr (LEV + 1 < PL.nlev) {
        row_level<LOGL, LEV>(ppc);
        row_levels<LOGL, LEV + 1>(ppc);
    }
}

template <int LOGL>
void row_plan_check() {
    constexpr int L = 1 << LOGL;
    row_levels<LOGL, 0>(1);
    if (small_ppc(LOGL) > 1) row_levels<LOGL, 0>(small_ppc(LOGL));
    // last level: 32-word groups read as 8 quads through the swizzle
    std::vector<int> seen(L, 0);
    for (int r = 0; r < L / 32; ++r)
        for (int c = 0; c < 8; ++c) {
            const int a = swz(r * 32 + 4 * c);
            CHECK(a % 4 == 0 && a >= 0 && a + 3 < L, "row L=%d quad", LOGL);
            for (int k = 0; k < 4; ++k)
                if (a + k >= 0 && a + k < L) seen[a + k]++;
        }
    for (int i = 0; i < L; ++i) CHECK(seen[i] == 1, "row L=%d last level word %d", LOGL, i);
}

template <int L1, int LEV>
void col_level() {
    using LV = ColLevel<L1, LEV>;
    constexpr int R = LV::R, TB = LV::TB, B = LV::B;
    constexpr int TASKS = (1 << L1) / R;
    for (int id = 0; id < TASKS; ++id) {
        const int blk = id / TB, o = id % TB;
        const int row0 = blk * B + o;
        for (int m = 0; m < R; ++m)
            CHECK((tile_row<L1>(row0) + tile_step<L1, TB>(m) == tile_row<L1>(row0 + TB * m)),
                  "col L1=%d lev=%d tile_step", L1, LEV);
        // tasks id (even) and id + 1 are on the two half-warps
        if (id % 2 == 0 && id + 1 < TASKS) {
            const int blk2 = (id + 1) / TB, o2 = (id + 1) % TB;
            const int row1 = blk2 * B + o2;
            for (int m = 0; m < R; ++m) {
                const int a = tile_row<L1>(row0 + TB * m), b = tile_row<L1>(row1 + TB * m);
                CHECK(((a - b) % 32 + 32) % 32 == 16, "col L1=%d lev=%d half-warp banks", L1, LEV);
            }
        }
        if (LEV + 1 < col_plan(L1).nlev)
            CHECK(LV::TWOFF + o * R + R - 1 < col_tw_entries(L1), "col L1=%d lev=%d twiddle", L1, LEV);
    }
}

template <int L1, int LEV>
void col_levels() {
    constexpr LevelPlan PL = col_plan(L1);
    if constexpr (LEV < PL.nlev) {
        col_level<L1, LEV>();
        col_levels<L1, LEV + 1>();
    }
}

// The staged column kernels' tile.
template <int L1>
void col_tile_check() {
    constexpr int n1 = 1 << L1;
    std::set<int> used;
    for (int r = 0; r < n1; ++r)
        for (int c = 0; c < kColTileCols; ++c) {
            const int a = tile_row<L1>(r) + c;
            CHECK((a >= 0 && a < col_tile_words(L1)), "col L1=%d out of tile", L1);
            CHECK(used.insert(a).second, "col L1=%d collision", L1);
        }
    // 16-byte quads of a row stay inside the row and 16-byte aligned
    for (int r = 0; r < n1; ++r) CHECK((tile_row<L1>(r) % 4 == 0), "col L1=%d quad alignment", L1);
    CHECK(col_smem_bytes(L1) <= 227 * 1024, "col L1=%d shared memory", L1);
    col_levels<L1, 0>();
}

// Rows leave a column pass in bit-reversed order, whatever its levels.
void col_order_check(int l1) {
    for (u32 s = 0; s < (1u << l1); ++s) CHECK(col_slot_to_k1(s, col_plan(l1), l1) == rev_bits(s, l1), "column order L1=%d", l1);
}

// The register column kernels (k_cold_fwd; k_cold_inv runs the same maps the
// other way): level 0's task o of column c reads rows o + R1 m and writes slot
// j to block j, the last level's task b reads its block and writes rows b R1 + m.
template <int L1>
void cold_check() {
    constexpr bool TWO = cold_two(L1);
    constexpr int n1 = 1 << L1, R0 = cold_r0(L1), R1 = cold_r1(L1), TC = cold_cols(L1), T = cold_threads(L1), BL = cold_block(L1);
    CHECK(R0 * R1 == n1 && (TWO || R1 == 1), "cold L1=%d radices", L1);
    CHECK(T % TC == 0 && T <= 1024, "cold L1=%d threads", L1);
    std::vector<int> in(n1, 0), out(n1, 0), wrote(cold_smem(L1) / 4 + 1, 0), read(cold_smem(L1) / 4 + 1, 0);
    for (int g = 0; g < T / TC; ++g)
        for (int o = g; o < R1; o += T / TC)
            for (int m = 0; m < R0; ++m) {
                in[o + R1 * m]++;
                if (!TWO) out[m]++;
                for (int c = 0; TWO && c < TC; ++c) {
                    const int a = o * TC + c + m * BL;
                    CHECK(a >= 0 && a < (int)(cold_smem(L1) / 4), "cold L1=%d tile", L1);
                    if (a >= 0 && a < (int)(cold_smem(L1) / 4)) wrote[a]++;
                }
                if (TWO) CHECK(o * R0 + m < col_tw_entries(L1) && (o * R0) % 2 == 0, "cold L1=%d twiddle", L1);
            }
    for (int g = 0; TWO && g < T / TC; ++g)
        for (int b = g; b < R0; b += T / TC)
            for (int m = 0; m < R1; ++m) {
                out[b * R1 + m]++;
                for (int c = 0; c < TC; ++c) {
                    const int a = b * BL + c + m * TC;
                    CHECK(a >= 0 && a < (int)(cold_smem(L1) / 4), "cold L1=%d tile", L1);
                    if (a >= 0 && a < (int)(cold_smem(L1) / 4)) read[a]++;
                }
            }
    for (int r = 0; r < n1; ++r) CHECK(in[r] == 1 && out[r] == 1, "cold L1=%d row %d", L1, r);
    for (size_t a = 0; a < wrote.size(); ++a) CHECK(wrote[a] == read[a] && wrote[a] <= 1, "cold L1=%d word %zu", L1, a);
    if (TWO && TC == 16) CHECK(BL % 32 == 16, "cold L1=%d half-warp banks", L1);
    CHECK((cold_smem(L1) + 1024) * cold_ctas(L1) <= 228 * 1024, "cold L1=%d shared memory", L1);
}

// The natural-order row kernel.
template <int L2>
void nat_check() {
    constexpr LevelPlan PL = nat_plan(L2);
    constexpr bool THREE = PL.nlev == 3;
    constexpr int n = 1 << L2, TPR = nat_row_threads(L2), S = nat_stride(L2), W = nat_words(L2);
    constexpr int R0 = 1 << PL.logr[0], TB0 = n / R0, R1 = THREE ? 1 << PL.logr[1] : 1, TB1 = TB0 / R1;
    constexpr int RL = 1 << PL.logr[PL.nlev - 1];
    CHECK(R0 * R1 * RL == n && TPR == TB0 && TB1 == RL, "nat L2=%d plan", L2);
    CHECK(nat_threads(L2) <= 1024 && nat_rows(L2) * W * 4 == (int)nat_smem(L2), "nat L2=%d shape", L2);
    CHECK((nat_smem(L2) + 1024) * nat_ctas(L2) <= 228 * 1024, "nat L2=%d shared memory", L2);
    std::vector<int> in(n, 0), out(n, 0), w0(W, 0), w1(W, 0), wl(W, 0), tw(nat_entries(L2), 0);
    auto hit = [&](std::vector<int>& v, int a) {
        CHECK(a >= 0 && a < (int)v.size(), "nat L2=%d index", L2);
        if (a >= 0 && a < (int)v.size()) v[a]++;
    };
    for (int t = 0; t < TPR; ++t)
        for (int k = 0; k < R0; ++k) {
            hit(in, t + TB0 * k);
            hit(w0, S * k + t);
            hit(tw, t + TB0 * k);
        }
    for (int t = 0; THREE && t < TPR; ++t)
        for (int id = t; id < R0 * TB1; id += TPR)
            for (int k = 0; k < R1; ++k) {
                hit(w1, S * (id / TB1) + id % TB1 + TB1 * k);
                if (id < TB1) hit(tw, n + id % TB1 + TB1 * k);
            }
    for (int t = 0; t < TPR; ++t)
        for (int id = t; id < n / RL; id += TPR)
            for (int k = 0; k < RL; ++k) {
                hit(wl, S * (id % R0) + RL * (id / R0) + k);
                hit(out, id + (n / RL) * k);
            }
    for (int i = 0; i < n; ++i) CHECK(in[i] == 1 && out[i] == 1, "nat L2=%d word %d", L2, i);
    for (int a = 0; a < W; ++a)
        CHECK(w0[a] <= 1 && wl[a] == w0[a] && (!THREE || w1[a] == w0[a]), "nat L2=%d exchange word %d", L2, a);
    for (size_t e = 0; e < tw.size(); ++e) CHECK(tw[e] == 1, "nat L2=%d twiddle %zu", L2, e);
}

// The row passes of a bivariate product: E bits of y and rows of 2^L2 words.
template <int E, int L2, int LEV>
void grid_levels() {
    constexpr int LT = grid_log(E, L2), N = 1 << LT;
    constexpr LevelPlan PL = row_plan(L2);
    if constexpr (LEV + 1 < PL.nlev) {
        using LV = SmallLevel<L2, LEV>;
        constexpr int R = LV::R, TB = LV::TB, B = LV::B;
        std::vector<int> seen(N, 0);
        for (int id = 0; id < N / R; ++id) {
            const int o = id % TB, base = (id / TB) * B + o, bs = swz(base);
            for (int m = 0; m < R; ++m) {
                const int a = swz_task<TB, B>(base, bs, m);
                CHECK((a == swz(base + TB * m) && a < N), "grid E=%d L2=%d lev=%d", E, L2, LEV);
                if (a >= 0 && a < N) seen[a]++;
                CHECK(LV::TWOFF + m * TB + o < plan_tw_entries(PL, L2), "grid E=%d L2=%d lev=%d twiddle", E, L2, LEV);
            }
        }
        for (int a = 0; a < N; ++a) CHECK(seen[a] == 1, "grid E=%d L2=%d lev=%d word %d", E, L2, LEV, a);
        grid_levels<E, L2, LEV + 1>();
    }
}

template <int E, int L2>
void grid_check() {
    constexpr int LT = grid_log(E, L2), N = 1 << LT;
    CHECK(grid_threads(LT) * 32 == N && (N * 4 + 1024) * grid_ctas(LT) <= 228 * 1024, "grid E=%d L2=%d shape", E, L2);
    if constexpr (E > 0) {
        // the level over y0: words 2^L2 apart, slot block (N / B) + blk's factors
        constexpr int R = 1 << E, TB = 1 << L2, B = TB << E;
        for (int slots = 1 << (LT - E - L2); slots <= 1 << 11; slots *= 2) {
            const int blocks = (int)(((long long)slots << (E + L2)) >> LT);
            CHECK(blocks >= 1 && ((long long)blocks << LT) == (long long)slots << (E + L2), "grid E=%d L2=%d blocks", E, L2);
            CHECK((blocks - 1) * (N / B) + N / B - 1 == slots - 1, "grid E=%d L2=%d slots", E, L2);
        }
        std::vector<int> seen(N, 0);
        for (int id = 0; id < N / R; ++id) {
            const int o = id % TB, base = (id / TB) * B + o, bs = swz(base);
            for (int m = 0; m < R; ++m) {
                const int a = swz_task<TB, B>(base, bs, m);
                CHECK((a == swz(base + TB * m) && a < N), "grid E=%d L2=%d leading level", E, L2);
                if (a >= 0 && a < N) seen[a]++;
            }
        }
        for (int a = 0; a < N; ++a) CHECK(seen[a] == 1, "grid E=%d L2=%d leading word %d", E, L2, a);
    }
    grid_levels<E, L2, 0>();
}

// G's row spectrum between the row kernels: quad c of 32-word group r at
// c * n2/8 + 4 r, a permutation of the row's quads; the lanes of a warp
// (consecutive r) cover one contiguous 512-byte run per quad index.
template <int L2>
void spectrum_layout_check() {
    constexpr int n2 = 1 << L2, G = n2 / 32;
    std::vector<int> hit(n2 / 4, 0);
    for (int r = 0; r < G; ++r)
        for (int c = 0; c < 8; ++c) {
            const int w = c * (n2 / 8) + 4 * r;
            CHECK((w % 4 == 0 && w + 3 < n2), "spectrum L2=%d quad in row", L2);
            if (w % 4 == 0 && w + 3 < n2) hit[w / 4]++;
            if (r % 32 != 0) CHECK(w == c * (n2 / 8) + 4 * (r - 1) + 4, "spectrum L2=%d warp run", L2);
        }
    for (int q = 0; q < n2 / 4; ++q) CHECK(hit[q] == 1, "spectrum L2=%d quad %d hit %d", L2, q, hit[q]);
}

template <int L2>
void row_tab_check() {
    using RT = RowTab<L2>;
    CHECK(RT::NA * RT::NB == RT::TB0, "rowtab L2=%d digits", L2);
    for (int o = 0; o < RT::TB0; ++o) {
        CHECK((o % RT::NA) + RT::NA * (o / RT::NA) == o, "rowtab L2=%d recompose", L2);
        for (int j = 0; j < RT::R0; ++j) {
            const int ia = (o % RT::NA) + j * RT::NA;
            const int ib = RT::R0 * RT::NA + o / RT::NA + j * RT::NB;
            CHECK(ia >= 0 && ia < RT::R0 * RT::NA, "rowtab L2=%d A index", L2);
            CHECK(ib >= RT::R0 * RT::NA && ib < RT::ENTRIES, "rowtab L2=%d B index", L2);
        }
    }
    // build loop (row_tab_build's decode): every table slot written once, the
    // power and twiddle read for it in bounds and of the slot's exponent
    std::vector<int> hit(RT::ENTRIES, 0);
    for (int q = 0; q < RT::ENTRIES; ++q) {
        const int j = q % RT::R0;
        int e, w, at;
        if (q < RT::R0 * RT::NA) { const int a = q / RT::R0; e = a; w = a; at = j * RT::NA + a; }
        else { const int k = (q - RT::R0 * RT::NA) / RT::R0; e = k * RT::NA; w = RT::NA + k; at = RT::R0 * RT::NA + j * RT::NB + k; }
        CHECK(at >= 0 && at < RT::ENTRIES, "rowtab L2=%d build slot", L2);
        if (at >= 0 && at < RT::ENTRIES) hit[at]++;
        CHECK(w >= 0 && w < RT::NPOW, "rowtab L2=%d build power", L2);
        CHECK(j * RT::TB0 + e < 1 << L2 && e < RT::TB0, "rowtab L2=%d build twiddle", L2);
        // the slot the level reads for (o, j) has exponent o mod NA, resp. NA (o div NA)
        if (q < RT::R0 * RT::NA) CHECK(at % RT::NA == e && at / RT::NA == j, "rowtab L2=%d A exponent", L2);
        else CHECK((at - RT::R0 * RT::NA) % RT::NB * RT::NA == e, "rowtab L2=%d B exponent", L2);
    }
    for (int i = 0; i < RT::ENTRIES; ++i) CHECK(hit[i] == 1, "rowtab L2=%d slot %d written %d times", L2, i, hit[i]);
    // shared memory of the split row kernels (+1 KiB reserved per CTA)
    const long long smem = (long long)(1 << L2) * 4 + (long long)RT::TABW * 8 + (long long)RT::NPOW * 4 + 2 * RT::R0 * 8;
    CHECK((RT::TABW * 8) % 16 == 0, "rowtab L2=%d table not a whole number of 16-byte copies", L2);
    CHECK((smem + 1024) * rowsplit_ctas(L2) <= 228 * 1024, "rowsplit L2=%d shared memory", L2);
}

void shoup_quot_check() {
    const u32 primes[] = {469762049u, 754974721u, 962592769u, 950009857u, 940572673u, 998244353u,
                          257u, 7681u, 12289u, 40961u, 1073479681u};
    unsigned long long st = 0x9E3779B97F4A7C15ull;
    for (u32 p : primes) {
        const double r = 4294967296.0 / (double)p;
        for (int k = 0; k < 200000; ++k) {
            st ^= st << 13; st ^= st >> 7; st ^= st << 17;
            u32 w = (u32)(st % p);
            if (k < 4) w = k < 2 ? (u32)k : p - (u32)(k - 1);
            const u32 want = (u32)(((unsigned long long)w << 32) / p);
            CHECK(shoup_quot_dev(w, p, r) == want, "shoup quotient p=%u w=%u", p, w);
        }
    }
}

template <int LOGL>
void latency_check(int cluster) {
    constexpr int L = 1 << LOGL;
    const LevelPlan pl = lat_plan(LOGL);
    std::vector<int> used((size_t)lat_words(LOGL), 0);
    for (int i = 0; i < L; ++i) {
        CHECK(lat_pad(i) < lat_words(LOGL), "latency L=%d pad out of range", LOGL);
        CHECK(used[(size_t)lat_pad(i)]++ == 0, "latency L=%d pad collides", LOGL);
    }
    int lb = LOGL, off = 0;
    for (int lev = 0; lev < pl.nlev; ++lev) {
        const int R = 1 << pl.logr[lev], B = 1 << lb, TB = B / R;
        std::vector<int> seen((size_t)L, 0);
        for (int id = 0; id < L / R; ++id) {
            const int o = id % TB, base = (id / TB) * B + o;
            for (int m = 0; m < R; ++m) {
                CHECK(base + TB * m < L, "latency L=%d level %d out of range", LOGL, lev);
                ++seen[(size_t)(base + TB * m)];
                if (lev + 1 < pl.nlev) CHECK(off + m * TB + o < lat_entries(LOGL), "latency L=%d twiddle", LOGL);
            }
        }
        for (int v : seen) CHECK(v == 1, "latency L=%d level %d coverage", LOGL, lev);
        if (lev + 1 < pl.nlev) off += B;
        lb -= pl.logr[lev];
    }
    CHECK(lb == 0 && pl.logr[pl.nlev - 1] == 3 && off == lat_entries(LOGL), "latency L=%d plan", LOGL);
    CHECK(lat_smem(LOGL, cluster) <= 227 * 1024, "latency L=%d shared memory", LOGL);
    CHECK(2 * L % lat_threads(LOGL) == 0, "latency L=%d load loop", LOGL);
    if (cluster > 1) {
        // words on their way home: block j's word i reaches CTA i / CH at j CH + i % CH
        const int CH = L / kClusterCtas;
        CHECK(2 * CH <= lat_threads(LOGL), "latency L=%d leading tasks", LOGL);
        std::vector<int> home((size_t)kClusterCtas * L, 0);
        for (int j = 0; j < kClusterCtas; ++j)
            for (int i = 0; i < L; ++i) {
                const int at = j * CH + i % CH;
                CHECK(at < L, "latency L=%d home", LOGL);
                ++home[(size_t)(i / CH) * L + at];
            }
        for (int v : home) CHECK(v == 1, "latency L=%d home coverage", LOGL);
    }
}

// The subproduct level kernel: the same blocks on its own CTA shape.
template <int LOGL>
void level_check() {
    constexpr int L = 1 << LOGL, T = level_threads(LOGL);
    latency_check<LOGL>(1);
    CHECK(2 * L % T == 0 && T <= 1024, "level L=%d load loop", LOGL);
    CHECK(T * level_ctas(LOGL) <= 2048 && level_ctas(LOGL) <= 32, "level L=%d residency", LOGL);
}

// latency_tables' exponents: entry (o, j) of a level of blocks of B = 2^lb
// words is (w^(2^(logn - lb)))^(+-o bitrev(j)), where the kernels read it.
template <int LOGL>
void latency_exponent_check(int logn) {
    const LevelPlan pl = lat_plan(LOGL);
    const u32 n = 1u << logn, ne = lat_entries(LOGL);
    const LatExponent ex{pl, LOGL, logn, (int)ne};
    auto both = [&](u32 fwd, u32 inv, u32 e, const char* what) {
        CHECK(ex(fwd) == e, "latency exponent L=%d %s", LOGL, what);
        CHECK(ex(inv) < n && (ex(inv) + e) % n == 0, "latency inverse exponent L=%d %s", LOGL, what);
    };
    u32 off = 0;
    int lb = LOGL;
    for (int lev = 0; lev + 1 < pl.nlev; ++lev) {
        const int r = pl.logr[lev];
        const u32 TB = 1u << (lb - r);
        for (u32 j = 0; j < 1u << r; ++j)
            for (u32 o = 0; o < TB; ++o)
                both(off + j * TB + o, ne + off + j * TB + o, (n >> lb) * o * rev_bits(j, r), "level");
        off += 1u << lb;
        lb -= r;
    }
    if (logn > LOGL)
        for (u32 j = 0; j < n >> LOGL; ++j)
            for (u32 o = 0; o < 1u << LOGL; ++o)
                both(2 * ne + (j << LOGL) + o, 2 * ne + n + (j << LOGL) + o, o * rev_bits(j, logn - LOGL), "lead");
}

// nat_slot_tables' exponents: slot s's W = w^k1(s): W^(TB m), then W^o.
template <int L2>
void slot_exponent_check(int l1) {
    const int r0 = 1 << nat_plan(L2).logr[0], tb = nat_row_threads(L2);
    const SlotExponent ex{col_plan(l1), l1, r0, tb};
    CHECK(r0 + tb == nat_slot_entries(L2) && r0 * tb == 1 << L2, "slot L2=%d entries", L2);
    for (u32 s = 0; s < 1u << l1; ++s) {
        const u32 k1 = col_slot_to_k1(s, col_plan(l1), l1), at = s * nat_slot_entries(L2);
        for (int m = 0; m < r0; ++m) CHECK(ex(at + m) == k1 * tb * m, "slot L2=%d factor", L2);
        for (int o = 0; o < tb; ++o) CHECK(ex(at + r0 + o) == k1 * o, "slot L2=%d task", L2);
        CHECK((long long)k1 * tb * (r0 - 1) < 1ll << (l1 + L2), "slot L2=%d exponent range", L2);
    }
}

int main() {
    latency_exponent_check<5>(5);
    latency_exponent_check<9>(9);
    latency_exponent_check<11>(11);
    latency_exponent_check<12>(12);
    latency_exponent_check<8>(12);
    latency_exponent_check<10>(14);
    latency_exponent_check<12>(16);
    slot_exponent_check<10>(5);
    slot_exponent_check<12>(5);
    slot_exponent_check<13>(5);
    slot_exponent_check<14>(10);
    slot_exponent_check<14>(11);
    level_check<5>();
    level_check<6>();
    level_check<7>();
    level_check<8>();
    level_check<9>();
    level_check<10>();
    level_check<11>();
    level_check<12>();
    latency_check<8>(16);
    latency_check<9>(16);
    latency_check<10>(16);
    latency_check<11>(16);
    latency_check<12>(16);
    row_plan_check<5>();
    row_plan_check<6>();
    row_plan_check<7>();
    row_plan_check<8>();
    row_plan_check<9>();
    row_plan_check<10>();
    row_plan_check<11>();
    row_plan_check<12>();
    row_plan_check<13>();
    row_plan_check<14>();
    for (int l1 = 1; l1 <= 11; ++l1) col_order_check(l1);
    col_tile_check<11>();
    cold_check<1>();
    cold_check<2>();
    cold_check<3>();
    cold_check<4>();
    cold_check<5>();
    cold_check<6>();
    cold_check<7>();
    cold_check<8>();
    cold_check<9>();
    cold_check<10>();
    nat_check<6>();
    nat_check<7>();
    nat_check<8>();
    nat_check<9>();
    nat_check<10>();
    nat_check<11>();
    nat_check<12>();
    nat_check<13>();
    nat_check<14>();
    grid_check<0, 6>();
    grid_check<0, 7>();
    grid_check<0, 8>();
    grid_check<0, 9>();
    grid_check<0, 10>();
    grid_check<0, 11>();
    grid_check<0, 12>();
    grid_check<0, 13>();
    grid_check<0, 14>();
    grid_check<1, 6>();
    grid_check<1, 7>();
    grid_check<1, 8>();
    grid_check<1, 9>();
    grid_check<1, 10>();
    grid_check<1, 11>();
    grid_check<1, 12>();
    grid_check<1, 13>();
    grid_check<2, 6>();
    grid_check<2, 7>();
    grid_check<2, 8>();
    grid_check<2, 9>();
    grid_check<2, 10>();
    grid_check<2, 11>();
    grid_check<2, 12>();
    spectrum_layout_check<6>();
    spectrum_layout_check<10>();
    spectrum_layout_check<11>();
    spectrum_layout_check<12>();
    spectrum_layout_check<13>();
    spectrum_layout_check<14>();
    row_tab_check<11>();
    row_tab_check<12>();
    row_tab_check<13>();
    row_tab_check<14>();
    shoup_quot_check();
    std::printf("%s: %d failures\n", failures ? "FAILED" : "OK", failures);
    return failures ? 1 : 0;
}
