// Natural-order transforms behind cumodp_fft_uni / cumodp_invfft_uni and
// the bivariate entry points.
//
// Reference behaviour: stockham_host / inverse_stockham_host
// (src/stockham.cu:479-503) compute X[j] = sum_i X[i] w^(ij) in natural
// order with the caller's root; bivariate_stockham_host
// (src/list_stockham.cu:1224-1245) computes the row-column 2-D DFT
// (DFT_m (x) I_n)(I_m (x) DFT_n) of a row-major 2^em x 2^en array.
//
// Here a transform of length <= 2^14 is one CTA's row (k_row_nat, natural
// order for free).  Longer 1-D transforms use the four-step split of the
// product path: a column pass (k_cold_fwd), the row pass (k_row_nat, SLOT),
// which applies w_n^(k1*c) and writes slot s as row k1(s) in natural order,
// and a tiled transpose.  The 2-D transform is the column pass plus the row
// pass with no inter-pass twiddle: its rows land directly in natural order.
#include <algorithm>
#include <cstring>
#include <vector>

#include "../../include/cumodp.h"
#include "product.cuh"
#include "row_natural.cuh"

namespace cmb {

__device__ __forceinline__ u32 seed_mont_at(const u32* __restrict__ seeds, int nlo, u32 e, u32 p, u32 pinv) {
    return mul_mont(__ldg(seeds + (e & 4095u)), __ldg(seeds + nlo + (e >> 12)), p, pinv);
}

// out[c * rows + r] = in[r * cols + c] for rows and cols multiples of 64:
// 64 x 64 tiles through shared memory, 16-byte loads and stores, 256
// threads (16 x 16, four 4-word groups each).
__global__ void __launch_bounds__(256) k_transpose64(const u32* __restrict__ in, u32* __restrict__ out, int rows,
                                                     int cols) {
    __shared__ u32 t[64][65];
    in += (size_t)blockIdx.z * rows * cols;  // transform blockIdx.z of a list
    out += (size_t)blockIdx.z * rows * cols;
    const size_t c0 = (size_t)blockIdx.x * 64, r0 = (size_t)blockIdx.y * 64;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const u32* src = in + r0 * cols + c0 + 4 * tx;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int rr = ty + 16 * k;
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(src + (size_t)rr * cols));
        t[rr][4 * tx] = v.x;
        t[rr][4 * tx + 1] = v.y;
        t[rr][4 * tx + 2] = v.z;
        t[rr][4 * tx + 3] = v.w;
    }
    __syncthreads();
    u32* dst = out + c0 * rows + r0 + 4 * tx;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int cc = ty + 16 * k;
        const uint4 v = make_uint4(t[4 * tx][cc], t[4 * tx + 1][cc], t[4 * tx + 2][cc], t[4 * tx + 3][cc]);
        *reinterpret_cast<uint4*>(dst + (size_t)cc * rows) = v;
    }
}

// out[c * rows + r] = in[r * cols + c]: 32 x 32 tiles through shared memory.
__global__ void k_transpose(const u32* __restrict__ in, u32* __restrict__ out, int rows, int cols) {
    __shared__ u32 t[32][33];
    in += (size_t)blockIdx.z * rows * cols;  // transform blockIdx.z of a list
    out += (size_t)blockIdx.z * rows * cols;
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int y = threadIdx.y; y < 32; y += blockDim.y)
        t[y][threadIdx.x] = in[(size_t)(r0 + y) * cols + c0 + threadIdx.x];
    __syncthreads();
    for (int y = threadIdx.y; y < 32; y += blockDim.y)
        out[(size_t)(c0 + y) * rows + r0 + threadIdx.x] = t[threadIdx.x][y];
}

// Direct DFT for n <= 32, one CTA of n threads per vector (vector b at
// offset b * n): out[j] = scale * sum x_i w^(ij).
__global__ void k_tiny_dft(const u32* __restrict__ x, u32* __restrict__ y, int n, u32 w, u32 p, u32 scale) {
    __shared__ u32 xs[32], pw[32];
    const int j = threadIdx.x;
    x += (size_t)blockIdx.x * n;
    y += (size_t)blockIdx.x * n;
    xs[j] = x[j] % p;
    u32 t = 1;
    for (int i = 0; i < j; ++i) t = (u32)(((u64)t * w) % p);
    pw[j] = t;
    __syncthreads();
    u64 acc = 0;
    for (int i = 0; i < n; ++i) acc = (acc + (u64)xs[i] * pw[(i * j) & (n - 1)]) % p;
    y[j] = (u32)((acc * scale) % p);
}

namespace {

// `rows` independent natural-order row transforms of 2^k words, 6 <= k <= 14
// (root: the transform's own, scale applied to every output): src row s to
// dst row s, or to row k1(s) when the rows are slots of a column pass of 2^l1.
template <int L2, bool SLOT>
int launch_row_nat_t(const RowNatArgs& a, int jobs, int dev, cudaStream_t st) {
    static DeviceOnce once;
    const int err = once(dev, [] { return allow_smem(k_row_nat<L2, SLOT>, nat_smem(L2)); });
    if (err != OK) return err;
    const u32 grid = (u32)(((u64)a.rows + nat_rows(L2) - 1) / nat_rows(L2));
    k_row_nat<L2, SLOT><<<dim3(grid, jobs), nat_threads(L2), nat_smem(L2), st>>>(a);
    return cuda_err(cudaGetLastError());
}
typedef int (*RowNatFn)(const RowNatArgs&, int, int, cudaStream_t);
const RowNatFn kRowNat[15] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                              launch_row_nat_t<6, false>, launch_row_nat_t<7, false>, launch_row_nat_t<8, false>,
                              launch_row_nat_t<9, false>, launch_row_nat_t<10, false>, launch_row_nat_t<11, false>,
                              launch_row_nat_t<12, false>, launch_row_nat_t<13, false>, launch_row_nat_t<14, false>};
// rows of a four-step transform (2^10 words and more)
const RowNatFn kRowSlot[15] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                               launch_row_nat_t<10, true>, launch_row_nat_t<11, true>, launch_row_nat_t<12, true>,
                               launch_row_nat_t<13, true>, launch_row_nat_t<14, true>};

int row_nat(const PrimeCtx& pc, const u32* src, u32* dst, long long rows, int k, u32 root, u32 scale, int l1, int dev,
            cudaStream_t st) {
    int err = OK;
    RowNatArgs A;
    memset(&A, 0, sizeof(A));
    A.tw = nat_tables(dev, pc.info.p, root, k, scale, &err);
    if (!A.tw) return err;
    A.pk = make_prime_k_for(pc.info, root, k);
    A.scaled = scale != 1u;
    A.l1 = l1;
    if (l1) A.colpl = col_plan(l1);
    cudaEvent_t e0;
    const bool tr = pass_timing_begin(st, &e0);
    for (long long r0 = 0; r0 < rows && err == OK; r0 += 1ll << 30) {  // one launch when l1 > 0
        A.src = src + (r0 << k);
        A.dst = dst + (r0 << k);
        A.rows = (u32)std::min<long long>(1ll << 30, rows - r0);
        err = kRowNat[k](A, 1, dev, st);
    }
    if (tr) pass_timing_end(st, "ntt_row", e0);
    return err;
}

// The rows of four-step transforms of 2^(l1 + l2) words with root `root`, and
// the transpose that follows: job t's rows (column-pass slots) at w1 + t n, its
// rows k1 in natural order at w2 + t n, its result at out + t n.
int rows_and_transpose(const PrimeCtx& pc, const u32* w1, u32* w2, u32* out, int l1, int l2, u32 root, u32 scale,
                       int jobs, int dev, cudaStream_t st) {
    int err = OK;
    const u32 p = pc.info.p, root_r = powmod_exact(root, 1ull << l1, p);
    RowNatArgs A;
    memset(&A, 0, sizeof(A));
    A.tw = nat_tables(dev, p, root_r, l2, scale, &err);
    A.slot = nat_slot_tables(dev, p, root, l1, l2, &err);
    if (!A.tw || !A.slot) return err;
    A.pk = make_prime_k_for(pc.info, root_r, l2);
    A.scaled = scale != 1u;
    A.l1 = l1;
    A.colpl = col_plan(l1);
    A.src = w1;
    A.dst = w2;
    A.rows = 1u << l1;
    A.job_stride = 1ll << (l1 + l2);
    cudaEvent_t e0;
    bool tr = pass_timing_begin(st, &e0);
    err = kRowSlot[l2](A, jobs, dev, st);
    if (tr) pass_timing_end(st, "ntt_row", e0);
    if (err != OK) return err;
    tr = pass_timing_begin(st, &e0);
    if (l1 >= 6)
        k_transpose64<<<dim3((1 << l2) / 64, (1 << l1) / 64, jobs), 256, 0, st>>>(w2, out, 1 << l1, 1 << l2);
    else
        k_transpose<<<dim3((1 << l2) / 32, (1 << l1) / 32, jobs), dim3(32, 8), 0, st>>>(w2, out, 1 << l1, 1 << l2);
    if (tr) pass_timing_end(st, "ntt_transpose", e0);
    return cuda_err(cudaGetLastError());
}

// w is a primitive 2^k-th root of unity mod p.
bool root_has_order(u32 w, int k, u32 p) {
    if (w == 0 || w >= p) return false;
    if (k == 0) return w == 1;
    return powmod_exact(w, 1ull << k, p) == 1 && powmod_exact(w, 1ull << (k - 1), p) == p - 1;
}

u32 inv_of(u32 a, u32 p) { return powmod_exact(a, p - 2, p); }

// Column pass of a single array (rows of n2 words, 2^l1 rows) into dst.
int column_pass(const PrimeCtx& pc, u32 root_c, int l1, int l2, const u32* src, long long len, u32* dst,
                int dev, cudaStream_t st, const LargeJob* djobs = nullptr, int njobs = 1) {
    int err = OK;
    const u32 p = pc.info.p;
    const Tw* twc = col_tables(dev, p, root_c, l1, &err);
    if (!twc) return err;
    LargeArgs A;
    memset(&A, 0, sizeof(A));
    A.pk = A.pkc = make_prime_k_for(pc.info, root_c, l1);
    A.twc = twc;
    A.twc_inv = plan_tw_entries(col_plan(l1), l1);
    A.l1 = l1;
    A.l2 = l2;
    A.colpl = col_plan(l1);
    A.job0 = LargeJob{src, nullptr, nullptr, (int)std::min<long long>(len, 1ll << 30), 0, 0, 0, dst, nullptr};
    A.jobs = djobs;  // a device job table (a list of transforms), or nullptr: job0
    A.njobs = njobs;
    if ((err = ensure_kernel_attrs(dev)) != OK) return err;
    launch_col_fwd1(A, njobs, st);
    return OK;
}

// First radix-2 (decimation-in-frequency) step of a transform of n = 2h
// words with root w: y0[j] = s (x[j] + x[j+h]) and y1[j] = s (x[j] - x[j+h])
// w^j for j < h, written over x_out[j] and x_out[j+h] (x_out may be x_in:
// each thread reads and writes the same four pairs).  Then the even outputs
// are DFT_h(y0; w^2) and the odd ones DFT_h(y1; w^2).  w^j * 2^32 is the
// Montgomery product of the seed-table words w^(j mod 4096) 2^32 and
// w^(4096 floor(j / 4096)) 2^32.  Inputs are any 32-bit words (reduced
// here); s = 1 (scaled = 0) or the inverse transform's 2^-k.
__global__ void __launch_bounds__(256) k_split_dif(const u32* x_in, u32* x_out, long long h,
                                                   const u32* __restrict__ seeds, int nlo, PrimeK pk, Tw s,
                                                   int scaled) {
    const u32 p = pk.p;
    const uint4* a4 = reinterpret_cast<const uint4*>(x_in);
    const uint4* b4 = reinterpret_cast<const uint4*>(x_in + h);
    uint4* y0 = reinterpret_cast<uint4*>(x_out);
    uint4* y1 = reinterpret_cast<uint4*>(x_out + h);
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < h / 4;
         q += (long long)gridDim.x * blockDim.x) {
        const uint4 av = a4[q], bv = b4[q];
        u32 a[4] = {av.x, av.y, av.z, av.w}, b[4] = {bv.x, bv.y, bv.z, bv.w}, u[4], v[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const u32 ra = red1(mul_shoup(a[t], 1u, pk.one_q, p), p);
            const u32 rb = red1(mul_shoup(b[t], 1u, pk.one_q, p), p);
            const u32 e = (u32)(4 * q + t);  // j < h <= 2^28
            const u32 wj = seed_mont_at(seeds, nlo, e, p, pk.pinv_neg);  // w^j 2^32, [0, 2p)
            u32 s0 = red1(ra + rb, p);
            u32 s1 = red1(mul_mont(ra - rb + p, wj, p, pk.pinv_neg), p);
            if (scaled) {
                s0 = red1(mul_shoup(s0, s.w, s.wq, p), p);
                s1 = red1(mul_shoup(s1, s.w, s.wq, p), p);
            }
            u[t] = s0;
            v[t] = s1;
        }
        y0[q] = make_uint4(u[0], u[1], u[2], u[3]);
        y1[q] = make_uint4(v[0], v[1], v[2], v[3]);
    }
}

// x[2m] = s0[m], x[2m+1] = s1[m] for m < h (the even and odd outputs of the
// split transform back in natural order).
__global__ void __launch_bounds__(256) k_interleave2(const u32* __restrict__ s0, const u32* __restrict__ s1,
                                                     u32* __restrict__ x, long long h) {
    const uint4* a4 = reinterpret_cast<const uint4*>(s0);
    const uint4* b4 = reinterpret_cast<const uint4*>(s1);
    uint4* x4 = reinterpret_cast<uint4*>(x);
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < h / 4;
         q += (long long)gridDim.x * blockDim.x) {
        const uint4 a = a4[q], b = b4[q];
        x4[2 * q] = make_uint4(a.x, b.x, a.y, b.y);
        x4[2 * q + 1] = make_uint4(a.z, b.z, a.w, b.w);
    }
}

}  // namespace

int ntt_natural_dev(const u32* x_in, u32* x_out, int k, u32 w, u32 p, bool inverse, cudaStream_t st);

namespace {

// A transform longer than the four-step kernels' 2^kMaxLog: one radix-2
// step over HBM (k_split_dif, which also applies the inverse's scaling),
// the two half-length transforms with root^2 (recursively), and the
// interleave of their outputs.  root is the transform's own root (already
// inverted for an inverse transform).
int ntt_split_dev(const PrimeCtx& pc, const u32* x_in, u32* x_out, int k, u32 root, u32 sc, cudaStream_t st) {
    int err = OK;
    const u32 p = pc.info.p;
    const long long n = 1ll << k, h = n / 2;
    const int dev = current_device();
    const u32* seeds = seed_tables(dev, p, root, k, &err);
    if (!seeds) return err ? err : OUT_OF_MEMORY;
    const Workspace S_space(dev, kWsSplitNtt + (k - kMaxLog - 1), (size_t)n * sizeof(u32), st, &err);
    u32* S = S_space.get();
    if (!S) return err;
    const int grid = 4 * sm_count(dev);
    k_split_dif<<<grid, 256, 0, st>>>(x_in, x_out, h, seeds, (int)std::min<long long>(n, 4096), pc.pk,
                                      tw_of(sc, p), sc != 1u);
    const u32 root2 = mulmod_exact(root, root, p);
    if ((err = ntt_natural_dev(x_out, S, k - 1, root2, p, false, st)) != OK) return err;
    if ((err = ntt_natural_dev(x_out + h, S + h, k - 1, root2, p, false, st)) != OK) return err;
    k_interleave2<<<grid, 256, 0, st>>>(S, S + h, x_out, h);
    return cuda_err(cudaGetLastError());
}

}  // namespace

// x_out = DFT(x_in) with root w (inverse: root w^-1 and scaling by 2^-k).
int ntt_natural_dev(const u32* x_in, u32* x_out, int k, u32 w, u32 p, bool inverse, cudaStream_t st) {
    int err = OK;
    const PrimeCtx* pc = prime_ctx(p, &err);
    if (!pc) return err;
    if (k < 0) return ASSUMPTION_ERROR;
    if (k >= 6 && (((uintptr_t)x_in | (uintptr_t)x_out) & 15)) return ASSUMPTION_ERROR;  // 16-byte rows
    if (k > pc->info.two_adic) return FFT_SIZE_TOO_LARGE;
    if (!root_has_order(w, k, p)) return ASSUMPTION_ERROR;
    if (k > kMaxSplitLog) return FFT_SIZE_TOO_LARGE;
    const int dev = current_device();
    const u32 root = inverse ? inv_of(w, p) : w;
    const u32 sc = inverse ? inv_of((u32)((1ull << k) % p), p) : 1u;
    if (k > kMaxLog) return ntt_split_dev(*pc, x_in, x_out, k, root, sc, st);
    if (k <= 5) {
        k_tiny_dft<<<1, 1 << k, 0, st>>>(x_in, x_out, 1 << k, root, p, sc);
        return cuda_err(cudaGetLastError());
    }
    if (k <= kMaxSmallLog) return row_nat(*pc, x_in, x_out, 1, k, root, sc, 0, dev, st);
    // the longest rows, and columns for the rest (no other split has been timed)
    const int l1 = std::max(5, k - kMaxRowLog), l2 = k - l1;
    const long long n = 1ll << k;
    const Workspace ws_space(dev, kWsNtt, (size_t)2 * n * sizeof(u32), st, &err);
    u32* ws = ws_space.get();
    if (!ws) return err;
    u32 *w1 = ws, *w2 = ws + n;
    const u32 root_c = powmod_exact(root, 1ull << l2, p);
    cudaEvent_t e0;
    const bool tr = pass_timing_begin(st, &e0);
    if ((err = column_pass(*pc, root_c, l1, l2, x_in, n, w1, dev, st)) != OK) return err;
    if (tr) pass_timing_end(st, "ntt_col", e0);
    return rows_and_transpose(*pc, w1, w2, x_out, l1, l2, root, sc, 1, dev, st);
}

namespace {

// m transforms of 2^k words (kMaxSmallLog < k <= kMaxLog), in place: the
// four-step passes of ntt_natural_dev, each launch covering up to
// min(2^16 - 1, 2^26 / 2^k) transforms (the column pass reads them from a
// job table, the row pass and the transpose take them from a grid
// dimension).  root is already inverted for an inverse transform.
int list_ntt_four_step(const PrimeCtx& pc, u32* x, long long m, int k, u32 root, u32 sc, cudaStream_t st) {
    int err = OK;
    const u32 p = pc.info.p;
    const int dev = current_device();
    const int l1 = std::max(5, k - kMaxRowLog), l2 = k - l1;
    const long long n = 1ll << k;
    const long long cm = std::min<long long>(m, std::max<long long>(1, std::min<long long>(65535, (1ll << 26) >> k)));
    const Workspace ws_space(dev, kWsNtt, (size_t)2 * cm * n * sizeof(u32), st, &err);
    u32* ws = ws_space.get();
    if (!ws) return err;
    const Workspace dj_space(dev, kWsListJobs, (size_t)cm * sizeof(LargeJob), st, &err);
    LargeJob* dj = dj_space.get<LargeJob>();
    if (!dj) return err;
    u32 *w1 = ws, *w2 = ws + cm * n;
    const u32 root_c = powmod_exact(root, 1ull << l2, p);
    std::vector<LargeJob> hj((size_t)cm);
    for (long long r0 = 0; r0 < m; r0 += cm) {
        const int cnt = (int)std::min(cm, m - r0);
        for (int t = 0; t < cnt; ++t)
            hj[t] = LargeJob{x + (r0 + t) * n, nullptr, nullptr, (int)n, 0, 0, 0, w1 + (long long)t * n, nullptr};
        // pageable source: staged before the call returns, so hj is free to refill
        cudaError_t e = cudaMemcpyAsync(dj, hj.data(), (size_t)cnt * sizeof(LargeJob), cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) return cuda_err(e);
        if ((err = column_pass(pc, root_c, l1, l2, nullptr, n, nullptr, dev, st, dj, cnt)) != OK) return err;
        if ((err = rows_and_transpose(pc, w1, w2, x + r0 * n, l1, l2, root, sc, cnt, dev, st)) != OK) return err;
    }
    return cuda_err(cudaGetLastError());
}

}  // namespace

// m independent natural-order transforms of length 2^k (row i at x + i 2^k),
// in place: the list transform I_m (x) DFT_n.
int list_ntt_dev(u32* x, long long m, int k, u32 w, u32 p, bool inverse, cudaStream_t st) {
    int err = OK;
    const PrimeCtx* pc = prime_ctx(p, &err);
    if (!pc) return err;
    if (m < 0 || k < 0) return ASSUMPTION_ERROR;
    if (k >= 6 && ((uintptr_t)x & 15)) return ASSUMPTION_ERROR;  // 16-byte rows
    if (m == 0) return OK;
    if (k > pc->info.two_adic) return FFT_SIZE_TOO_LARGE;
    if (!root_has_order(w, k, p)) return ASSUMPTION_ERROR;
    const u32 root = inverse ? inv_of(w, p) : w;
    const u32 sc = inverse ? inv_of((u32)((1ull << k) % p), p) : 1u;
    if (k <= 5) {
        for (long long r0 = 0; r0 < m; r0 += 65535) {
            const unsigned nb = (unsigned)std::min<long long>(65535, m - r0);
            k_tiny_dft<<<nb, 1 << k, 0, st>>>(x + (r0 << k), x + (r0 << k), 1 << k, root, p, sc);
        }
        return cuda_err(cudaGetLastError());
    }
    if (k <= kMaxSmallLog) return row_nat(*pc, x, x, m, k, root, sc, 0, current_device(), st);
    if (k <= kMaxLog) return list_ntt_four_step(*pc, x, m, k, root, sc, st);
    for (long long r = 0; r < m; ++r)
        if ((err = ntt_natural_dev(x + (r << k), x + (r << k), k, w, p, inverse, st)) != OK) return err;
    return OK;
}

namespace {

// out[c * rows + r] = in[r * cols + c]: 32 x 32 tiles through shared memory,
// bounds-checked.  blockIdx.x runs over the longer side (rows_on_x), so any
// shape with rows * cols <= 2^30 fits the grid (the shorter side is then at
// most 2^15 long).
__global__ void k_transpose_long(const u32* __restrict__ in, u32* __restrict__ out, long long rows, long long cols,
                                 int rows_on_x) {
    __shared__ u32 t[32][33];
    const long long r0 = 32ll * (rows_on_x ? blockIdx.x : blockIdx.y);
    const long long c0 = 32ll * (rows_on_x ? blockIdx.y : blockIdx.x);
    for (int y = threadIdx.y; y < 32; y += blockDim.y)
        if (r0 + y < rows && c0 + threadIdx.x < cols) t[y][threadIdx.x] = in[(r0 + y) * cols + c0 + threadIdx.x];
    __syncthreads();
    for (int y = threadIdx.y; y < 32; y += blockDim.y)
        if (c0 + y < cols && r0 + threadIdx.x < rows) out[(c0 + y) * rows + r0 + threadIdx.x] = t[threadIdx.x][y];
}

void transpose_long(const u32* in, u32* out, long long rows, long long cols, cudaStream_t st) {
    const unsigned tr = (unsigned)((rows + 31) / 32), tc = (unsigned)((cols + 31) / 32);
    const bool rx = tr >= tc;
    k_transpose_long<<<rx ? dim3(tr, tc) : dim3(tc, tr), dim3(32, 8), 0, st>>>(in, out, rows, cols, rx ? 1 : 0);
}

// A 2-D transform past the fused path's limits (columns longer than
// 2^kMaxColLog or rows longer than 2^kMaxRowLog): the rows as a list
// transform in place, then the columns as a list transform of the
// transposed array, transposed back.  Each list transform applies its own
// inverse scaling (2^-en, 2^-em).
int bivariate_general(u32* x, int em, u32 wm, int en, u32 wn, u32 p, bool inverse, cudaStream_t st) {
    int err = OK;
    if (em + en > 30) return FFT_SIZE_TOO_LARGE;
    const long long rows = 1ll << em, cols = 1ll << en;
    if ((err = list_ntt_dev(x, rows, en, wn, p, inverse, st)) != OK) return err;
    if (em == 0) return OK;
    const Workspace t_space(current_device(), kWsBivT, (size_t)(rows * cols) * sizeof(u32), st, &err);
    u32* t = t_space.get();
    if (!t) return err;
    transpose_long(x, t, rows, cols, st);
    if ((err = list_ntt_dev(t, cols, em, wm, p, inverse, st)) != OK) return err;
    transpose_long(t, x, cols, rows, st);
    return cuda_err(cudaGetLastError());
}

}  // namespace

// 2-D DFT of a row-major 2^em x 2^en array, in place.
int bivariate_dev(u32* x, int em, u32 wm, int en, u32 wn, u32 p, bool inverse, cudaStream_t st) {
    int err = OK;
    const PrimeCtx* pc = prime_ctx(p, &err);
    if (!pc) return err;
    if (em < 0 || en < 0) return ASSUMPTION_ERROR;
    if ((uintptr_t)x & 15) return ASSUMPTION_ERROR;  // 16-byte rows
    if (em > pc->info.two_adic || en > pc->info.two_adic) return FFT_SIZE_TOO_LARGE;
    if (!root_has_order(wm, em, p) || !root_has_order(wn, en, p)) return ASSUMPTION_ERROR;
    if (en < 6) return FFT_SIZE_TOO_SMALL;
    if (en > kMaxRowLog || em > kMaxColLog) return bivariate_general(x, em, wm, en, wn, p, inverse, st);
    const int dev = current_device();
    const u32 rm = inverse ? inv_of(wm, p) : wm, rn = inverse ? inv_of(wn, p) : wn;
    const u32 sc = inverse ? inv_of((u32)((1ull << (em + en)) % p), p) : 1u;
    const long long total = 1ll << (em + en);
    if (em == 0) return row_nat(*pc, x, x, 1, en, rn, sc, 0, dev, st);
    const Workspace w1_space(dev, kWsNtt, (size_t)total * sizeof(u32), st, &err);
    u32* w1 = w1_space.get();
    if (!w1) return err;
    if ((err = column_pass(*pc, rm, em, en, x, total, w1, dev, st)) != OK) return err;
    return row_nat(*pc, w1, x, 1ll << em, en, rn, sc, em, dev, st);
}

// a[i] = a[i] * b[i] mod p (inputs in [0, p)): a Montgomery product
// (a b 2^-32) times r2 = 2^64 mod p by a second one, then one reduction.
__global__ void k_pointwise_mod(u32* __restrict__ a, const u32* __restrict__ b, long long n, u32 p, u32 pinv_neg,
                                u32 r2) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        a[i] = red1(mul_mont(mul_mont(a[i], b[i], p, pinv_neg), r2, p, pinv_neg), p);
}

// dst (2^ey2 rows of 2^ex2) = src (ny1 rows of nx1) zero-padded, reduced mod p.
__global__ void k_expand2(const u32* __restrict__ src, int nx1, int ny1, u32* __restrict__ dst, int ex2, int ey2,
                          u32 p) {
    const long long total = 1ll << (ex2 + ey2);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long y = i >> ex2, x = i & ((1ll << ex2) - 1);
        dst[i] = (x < nx1 && y < ny1) ? src[y * nx1 + x] % p : 0u;
    }
}

// dst (ny1 rows of nx1) = the top-left corner of src (rows of 2^ex2).
__global__ void k_extract2(const u32* __restrict__ src, int ex2, u32* __restrict__ dst, int nx1, int ny1) {
    const long long total = (long long)nx1 * ny1;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long y = i / nx1, x = i % nx1;
        dst[i] = src[(y << ex2) + x];
    }
}

int grid_for(long long n) { return (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, 148 * 16)); }

// f <- f * g mod (x^n - 1, p), n = 2^e, for the lengths the product kernels
// do not cover (e < 5 or e > 25): natural-order transforms of f (in place)
// and of g (into workspace, so g is left as it is), the pointwise product and
// the inverse transform of f.
int cyclic_mul_compose(u32* f, const u32* g, int e, u32 p, cudaStream_t st) {
    int err = OK;
    const PrimeCtx* pc = prime_ctx(p, &err);
    if (!pc) return err;
    const long long n = 1ll << e;
    const u32 w = canonical_root(*pc, e);
    const Workspace gt_space(current_device(), kWsCyclic, (size_t)n * sizeof(u32), st, &err);
    u32* gt = gt_space.get();
    if (!gt) return err;
    if ((err = ntt_natural_dev(g, gt, e, w, p, false, st)) != OK) return err;
    if ((err = ntt_natural_dev(f, f, e, w, p, false, st)) != OK) return err;
    k_pointwise_mod<<<grid_for(n), 256, 0, st>>>(f, gt, n, p, pc->info.pinv_neg, pc->info.r2);
    if ((err = cuda_err(cudaGetLastError())) != OK) return err;
    return ntt_natural_dev(f, f, e, w, p, true, st);
}

// F <- DFT^-1(DFT F * DFT G) on a 2^em x 2^en row-major grid (rows: y, of
// length 2^en in x): the 2-D cyclic convolution, i.e. the bivariate product
// when both operands are zero-padded to the product's size.  Grids of up to
// 2^13 rows run as the three passes of a long product (grid_mul_dev).
// Otherwise: row transforms,
// a transpose, column transforms (as rows) give both spectra in transposed
// order; the pointwise product and the inverse steps run in that order, so
// nothing is permuted back before the last transpose.  G is overwritten.
int bivariate_mul_dev(u32* F, u32* G, int em, int en, u32 p, cudaStream_t st) {
    int err = OK;
    const PrimeCtx* pc = prime_ctx(p, &err);
    if (!pc) return err;
    if (em < 0 || en < 0) return ASSUMPTION_ERROR;
    if ((em >= 6 || en >= 6) && (((uintptr_t)F | (uintptr_t)G) & 15)) return ASSUMPTION_ERROR;  // 16-byte rows
    if (em > pc->info.two_adic || en > pc->info.two_adic || em + en > 30) return FFT_SIZE_TOO_LARGE;
    const long long m = 1ll << em, n = 1ll << en, total = m * n;
    const u32 wm = em ? canonical_root(*pc, em) : 1u, wn = en ? canonical_root(*pc, en) : 1u;
    int l1, e;
    if (grid_split(em, en, &l1, &e)) {
        // needs two grids of workspace; without them the paths below, which
        // leave the operands as they are until their own workspace is there
        err = grid_mul_dev(F, G, em, en, p, st);
        if (err != OUT_OF_MEMORY) return err;
    }
    if (en >= 6 && en <= kMaxRowLog && em <= kMaxColLog) {
        // one row, a grid of less than 2^11 words, or no room for two grids
        if ((err = bivariate_dev(F, em, wm, en, wn, p, false, st)) != OK) return err;
        if ((err = bivariate_dev(G, em, wm, en, wn, p, false, st)) != OK) return err;
        k_pointwise_mod<<<grid_for(total), 256, 0, st>>>(F, G, total, p, pc->info.pinv_neg, pc->info.r2);
        if ((err = bivariate_dev(F, em, wm, en, wn, p, true, st)) != OK) return err;
        return cuda_err(cudaGetLastError());
    }
    const int dev = current_device();
    const long long tpad = (total + 3) & ~3ll;  // 16-byte aligned halves
    const Workspace ws_space(dev, kWsBiv, (size_t)2 * tpad * sizeof(u32), st, &err);
    u32* ws = ws_space.get();
    if (!ws) return err;
    u32 *W1 = ws, *W2 = ws + tpad;
    u32* src[2] = {F, G};
    u32* spec[2] = {W1, W2};
    for (int o = 0; o < 2; ++o) {
        if ((err = list_ntt_dev(src[o], m, en, wn, p, false, st)) != OK) return err;
        transpose_long(src[o], spec[o], m, n, st);
        if ((err = list_ntt_dev(spec[o], n, em, wm, p, false, st)) != OK) return err;
    }
    k_pointwise_mod<<<grid_for(total), 256, 0, st>>>(W1, W2, total, p, pc->info.pinv_neg, pc->info.r2);
    if ((err = list_ntt_dev(W1, n, em, wm, p, true, st)) != OK) return err;
    transpose_long(W1, F, n, m, st);
    if ((err = list_ntt_dev(F, m, en, wn, p, true, st)) != OK) return err;
    return cuda_err(cudaGetLastError());
}

// Bivariate product of (nx, ny)-dense operands (coefficient of x^i y^j at
// j * nx + i), device buffers: H gets (nxf + nxg - 1) x (nyf + nyg - 1).
int bivariate_product_dev(const u32* F, int nxf, int nyf, const u32* G, int nxg, int nyg, u32* H, u32 p,
                          cudaStream_t st) {
    int err = OK;
    const long long lx = (long long)nxf + nxg - 1, ly = (long long)nyf + nyg - 1;
    int ex = 0, ey = 0;
    while ((1ll << ex) < lx) ++ex;
    while ((1ll << ey) < ly) ++ey;
    if (ex + ey > 30) return FFT_SIZE_TOO_LARGE;
    const long long total = 1ll << (ex + ey);
    const long long tpad = (total + 3) & ~3ll;  // 16-byte aligned halves
    const Workspace ws_space(current_device(), kWsBivHost, (size_t)2 * tpad * sizeof(u32), st, &err);
    u32* ws = ws_space.get();
    if (!ws) return err;
    u32 *F2 = ws, *G2 = ws + tpad;
    k_expand2<<<grid_for(total), 256, 0, st>>>(F, nxf, nyf, F2, ex, ey, p);
    k_expand2<<<grid_for(total), 256, 0, st>>>(G, nxg, nyg, G2, ex, ey, p);
    if ((err = bivariate_mul_dev(F2, G2, ey, ex, p, st)) != OK) return err;
    k_extract2<<<grid_for(lx * ly), 256, 0, st>>>(F2, ex, H, (int)lx, (int)ly);
    return cuda_err(cudaGetLastError());
}

}  // namespace cmb

using namespace cmb;

namespace {

cumodp_err host_ntt(sfixn* X, sfixn n, sfixn k, sfixn w, sfixn p, bool inverse) {
    int cnt = 0;
    if (cudaGetDeviceCount(&cnt) != cudaSuccess || cnt == 0) {
        cudaGetLastError();
        return CUMODP_NO_CUDA_DEVICE;
    }
    if (!X || k < 0 || k > 30 || n != (sfixn)(1u << k) || p <= 0) return CUMODP_ASSUMPTION_ERROR;
    std::lock_guard<std::mutex> g(lib_mutex());
    const int dev = current_device();
    cudaStream_t st = lib_stream(dev);
    int err = OK;
    const Workspace d_space(dev, kWsStage, (size_t)n * sizeof(u32), st, &err);
    u32* d = d_space.get();
    if (!d) return (cumodp_err)err;
    cudaError_t ce = cudaMemcpyAsync(d, X, (size_t)n * 4, cudaMemcpyHostToDevice, st);
    if (ce != cudaSuccess) return (cumodp_err)cuda_err(ce);
    err = ntt_natural_dev(d, d, k, (u32)w, (u32)p, inverse, st);
    if (err != OK) {
        cudaStreamSynchronize(st);
        return (cumodp_err)err;
    }
    ce = cudaMemcpyAsync(X, d, (size_t)n * 4, cudaMemcpyDeviceToHost, st);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
    return (cumodp_err)cuda_err(ce);
}

cumodp_err host_bivariate(sfixn* X, sfixn em, sfixn wm, sfixn en, sfixn wn, sfixn p, bool inverse) {
    int cnt = 0;
    if (cudaGetDeviceCount(&cnt) != cudaSuccess || cnt == 0) {
        cudaGetLastError();
        return CUMODP_NO_CUDA_DEVICE;
    }
    if (!X || em < 0 || en < 0 || em + en > 30 || p <= 0) return CUMODP_ASSUMPTION_ERROR;
    std::lock_guard<std::mutex> g(lib_mutex());
    const int dev = current_device();
    cudaStream_t st = lib_stream(dev);
    const size_t total = (size_t)1 << (em + en);
    int err = OK;
    const Workspace d_space(dev, kWsStage, total * sizeof(u32), st, &err);
    u32* d = d_space.get();
    if (!d) return (cumodp_err)err;
    cudaError_t ce = cudaMemcpyAsync(d, X, total * 4, cudaMemcpyHostToDevice, st);
    if (ce != cudaSuccess) return (cumodp_err)cuda_err(ce);
    err = bivariate_dev(d, em, (u32)wm, en, (u32)wn, (u32)p, inverse, st);
    if (err != OK) {
        cudaStreamSynchronize(st);
        return (cumodp_err)err;
    }
    ce = cudaMemcpyAsync(X, d, total * 4, cudaMemcpyDeviceToHost, st);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
    return (cumodp_err)cuda_err(ce);
}

}  // namespace

extern "C" {

cumodp_err cumodp_fft_uni_dev(sfixn* X, sfixn n, sfixn k, sfixn w, sfixn p, int inverse, void* stream) {
    int cnt = 0;
    if (cudaGetDeviceCount(&cnt) != cudaSuccess || cnt == 0) {
        cudaGetLastError();
        return CUMODP_NO_CUDA_DEVICE;
    }
    if (!X || k < 0 || k > 30 || n != (sfixn)(1u << k) || p <= 0) return CUMODP_ASSUMPTION_ERROR;
    std::lock_guard<std::mutex> g(lib_mutex());
    cudaStream_t st = stream ? (cudaStream_t)stream : lib_stream(current_device());
    int e = ntt_natural_dev((const u32*)X, (u32*)X, k, (u32)w, (u32)p, inverse != 0, st);
    if (e == OK && !stream) e = cuda_err(cudaStreamSynchronize(st));
    return (cumodp_err)e;
}

cumodp_err cumodp_fft_bivariate_dev(sfixn* X, sfixn em, sfixn wm, sfixn en, sfixn wn, sfixn p, int inverse,
                                    void* stream) {
    int cnt = 0;
    if (cudaGetDeviceCount(&cnt) != cudaSuccess || cnt == 0) {
        cudaGetLastError();
        return CUMODP_NO_CUDA_DEVICE;
    }
    if (!X || em < 0 || en < 0 || em + en > 30 || p <= 0) return CUMODP_ASSUMPTION_ERROR;
    std::lock_guard<std::mutex> g(lib_mutex());
    cudaStream_t st = stream ? (cudaStream_t)stream : lib_stream(current_device());
    int e = bivariate_dev((u32*)X, em, (u32)wm, en, (u32)wn, (u32)p, inverse != 0, st);
    if (e == OK && !stream) e = cuda_err(cudaStreamSynchronize(st));
    return (cumodp_err)e;
}

cumodp_err cumodp_list_fft_dev(sfixn* X, sfixn m, sfixn k, sfixn w, sfixn p, int inverse, void* stream) {
    int cnt = 0;
    if (cudaGetDeviceCount(&cnt) != cudaSuccess || cnt == 0) {
        cudaGetLastError();
        return CUMODP_NO_CUDA_DEVICE;
    }
    if (!X || m < 0 || k < 0 || k > 30 || p <= 0) return CUMODP_ASSUMPTION_ERROR;
    std::lock_guard<std::mutex> g(lib_mutex());
    cudaStream_t st = stream ? (cudaStream_t)stream : lib_stream(current_device());
    int e = list_ntt_dev((u32*)X, m, k, (u32)w, (u32)p, inverse != 0, st);
    if (e == OK && !stream) e = cuda_err(cudaStreamSynchronize(st));
    return (cumodp_err)e;
}

cumodp_err cumodp_bivariate_mul_dev(sfixn em, sfixn en, sfixn* F, sfixn* G, sfixn p, void* stream) {
    int cnt = 0;
    if (cudaGetDeviceCount(&cnt) != cudaSuccess || cnt == 0) {
        cudaGetLastError();
        return CUMODP_NO_CUDA_DEVICE;
    }
    if (!F || !G || em < 0 || en < 0 || p <= 0) return CUMODP_ASSUMPTION_ERROR;
    std::lock_guard<std::mutex> g(lib_mutex());
    cudaStream_t st = stream ? (cudaStream_t)stream : lib_stream(current_device());
    int e = bivariate_mul_dev((u32*)F, (u32*)G, em, en, (u32)p, st);
    if (e == OK && !stream) e = cuda_err(cudaStreamSynchronize(st));
    return (cumodp_err)e;
}

cumodp_err cumodp_bivariate_mul(sfixn nxf, sfixn nyf, const sfixn* F, sfixn nxg, sfixn nyg, const sfixn* G,
                                sfixn* H, sfixn p) {
    int cnt = 0;
    if (cudaGetDeviceCount(&cnt) != cudaSuccess || cnt == 0) {
        cudaGetLastError();
        return CUMODP_NO_CUDA_DEVICE;
    }
    if (!F || !G || !H || nxf <= 0 || nyf <= 0 || nxg <= 0 || nyg <= 0 || p <= 0) return CUMODP_ASSUMPTION_ERROR;
    const long long nf = (long long)nxf * nyf, ng = (long long)nxg * nyg;
    const long long nh = ((long long)nxf + nxg - 1) * ((long long)nyf + nyg - 1);
    if (nh > (1ll << 30)) return CUMODP_FFT_SIZE_TOO_LARGE;
    std::lock_guard<std::mutex> g(lib_mutex());
    const int dev = current_device();
    cudaStream_t st = lib_stream(dev);
    int err = OK;
    const Workspace d_space(dev, kWsStage, (size_t)(nf + ng + nh) * sizeof(u32), st, &err);
    u32* d = d_space.get();
    if (!d) return (cumodp_err)err;
    cudaError_t ce = cudaMemcpyAsync(d, F, nf * 4, cudaMemcpyHostToDevice, st);
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(d + nf, G, ng * 4, cudaMemcpyHostToDevice, st);
    if (ce != cudaSuccess) return (cumodp_err)cuda_err(ce);
    err = bivariate_product_dev(d, nxf, nyf, d + nf, nxg, nyg, d + nf + ng, (u32)p, st);
    if (err != OK) {
        cudaStreamSynchronize(st);
        return (cumodp_err)err;
    }
    ce = cudaMemcpyAsync(H, d + nf + ng, nh * 4, cudaMemcpyDeviceToHost, st);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
    return (cumodp_err)cuda_err(ce);
}

cumodp_err cumodp_fft_uni(sfixn* X, sfixn n, sfixn k, sfixn w, sfixn p) { return host_ntt(X, n, k, w, p, false); }

cumodp_err cumodp_invfft_uni(sfixn* X, sfixn n, sfixn k, sfixn w, sfixn p) { return host_ntt(X, n, k, w, p, true); }

cumodp_err cumodp_fft_bivariate(sfixn* X, sfixn em, sfixn wm, sfixn en, sfixn wn, sfixn p) {
    return host_bivariate(X, em, wm, en, wn, p, false);
}

cumodp_err cumodp_invfft_bivariate(sfixn* X, sfixn em, sfixn wm, sfixn en, sfixn wn, sfixn p) {
    return host_bivariate(X, em, wm, en, wn, p, true);
}

}  // extern "C"
