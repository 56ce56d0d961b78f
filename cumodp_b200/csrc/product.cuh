// Host-side product dispatch shared by the C entry points.
#pragma once
#include "large_product.cuh"
#include "latency_product.cuh"
#include "runtime.cuh"

namespace cmb {

constexpr int kMinLog = 5;        // smallest transform: one radix-32 row
constexpr int kMaxSmallLog = 14;  // largest single-CTA product (2 x 64 KiB of shared memory)
constexpr int kMaxColLog = 11;    // 16-column tile of 2^11 rows = 136 KiB of shared memory
constexpr int kMaxRowLog = 14;
constexpr int kMinRowLog = 6;
constexpr int kMaxLog = 25;        // largest transform of the three-pass kernels (2^11 x 2^14)
constexpr int kMaxSplitLog = 29;   // longer single products and transforms, up to the prime's 2-adic
                                   // order (at most 29 for p < 2^30), are split into 2^25 pieces
constexpr int kDefaultColLog = 10;  // column length of the default split (rows of 2^14)

// workspace slots (runtime.cuh: workspace)
enum WsSlot { kWsSingle = 0, kWsBatch = 1, kWsStage = 2, kWsNtt = 3, kWsTwoConv = 4, kWsServer = 5,
              kWsBiv = 6, kWsBivHost = 7, kWsBig = 8, kWsSplitProd = 9, kWsSplitIn = 10,
              kWsSplitNtt = 11 /* + (k - kMaxLog - 1) for a 2^k transform: 11..14 */, kWsBivT = 15,
              kWsListJobs = 16, kWsCyclic = 17 };
// pinned host staging slots (runtime.cuh: pinned_workspace)
enum PinSlot { kPinTwoConv = 0, kPinMul = 1 };

// SMs of device dev (cached per device).
int sm_count(int dev);

// Transform length log2 for a product of la and lb coefficients.
int product_logn(long long la, long long lb);
// Default row length log2 of the three-pass split.
int default_row_log(int logn);

int small_args(const PrimeCtx& pc, u32 root, int logn, int dev, SmallArgs* a);
int large_args(const PrimeCtx& pc, u32 root_n, int logn, int l2, int dev, LargeArgs* a);
// The forward column pass of every job's two operands; that of operand a alone;
// the inverse column pass.
void launch_col_fwd(const LargeArgs& a, int njobs, cudaStream_t st);
void launch_col_fwd1(const LargeArgs& a, int njobs, cudaStream_t st);
void launch_col_inv(const LargeArgs& a, int njobs, cudaStream_t st);
void launch_small(int logn, const SmallArgs& a, int njobs, cudaStream_t st);
void launch_large(const LargeArgs& a, int njobs, cudaStream_t st);

// A single product of transform length 2^logn (kMinLog <= logn <=
// kMaxLatencyLog) in one launch (latency_product.cuh); *launched = false when
// the device cannot run it (no room for a cluster of 16 CTAs) and the caller
// takes the other kernels.  The limit is what a cluster's shared memory holds;
// at 2^16 the one launch takes 11.5 us and the three-pass kernels 14.8.
constexpr int kMaxLatencyLog = 16;
int latency_mul(const PrimeCtx& pc, int logn, int dev, const ProdJob& job, cudaStream_t st, bool* launched);
// Whether it will run there (its tables are ready then).
int latency_usable(const PrimeCtx& pc, int logn, int dev, bool* usable);
// Products of the same lengths mod np (3 or 4) primes: prime r's operands at
// a + r astride, b + r bstride, its la + lb - 1 residues at h + r hstride.
int latency_mul_primes(const u32* primes, int np, int dev, const u32* a, int la, long long astride, const u32* b, int lb,
                       long long bstride, u32* h, long long hstride, cudaStream_t st, bool* launched);
// The same for two signed 64-bit operands mod np (2 or 3) primes in one
// launch: prime r's la + lb - 1 residues at h + r (la + lb - 1).  *launched =
// false past 2^kMaxLatencyLog too.
int latency_mul_i64(const u32* primes, int np, int dev, const long long* a, int la, const long long* b, int lb, u32* h,
                    cudaStream_t st, bool* launched);

// One level of a subproduct tree, 2l <= 2^kMaxLevelLog (k_monic_level): the
// npairs products of consecutive monic polynomials of degree l.  Longer levels
// have few pairs for their size and run as batches (2^13 words are two
// operands and twiddles of more than one CTA's shared memory).
constexpr int kMaxLevelLog = 12;
int monic_level_dev(const PrimeCtx& pc, int l, int npairs, const u32* in, u32* out, cudaStream_t st);

// Sets the shared-memory limits of every product kernel on the current device
// dev, once (must run before the first launch there).
int ensure_kernel_attrs(int dev);

// Batched products on caller-owned buffers, direct launches (batch.cu).
size_t direct_ws_words(int count, const long long* la, const long long* lb);
size_t direct_job_bytes(int count);
// allow_tuning: a size class seen for the first time may be autotuned
// (synchronous timing runs); otherwise cached choices or the default split.
int direct_batch(int count, const u32* const* a, const long long* la, const u32* const* b, const long long* lb,
                 u32* const* h, const long long* lh, u32 p, u32* ws, void* djobs, void* hjobs,
                 cudaStream_t st, bool allow_tuning);

// Device words of workspace a single product of transform length 2^logn
// takes (mul_dev), beside its operands and result.
size_t mul_ws_words(int logn);

// h[0..lh) = a[0..la) * b[0..lb) mod p on device pointers, on stream st.
int mul_dev(const u32* a, long long la, const u32* b, long long lb, u32* h, long long lh, u32 p,
            cudaStream_t st);

// Whether the bivariate product of 2^em x 2^en grids runs on the three-pass
// kernels (grid_product.cuh): columns of 2^l1 rows, the other e bits of y in
// the row passes.
bool grid_split(int em, int en, int* l1, int* e);
// F <- the 2-D cyclic convolution of F and G (grids within grid_split's range,
// 16-byte aligned; em and en within p's 2-adic order).
int grid_mul_dev(u32* F, u32* G, int em, int en, u32 p, cudaStream_t st);

// f <- f * g mod (x^(2^e) - 1, p), the length-2^e cyclic convolution, on
// device arrays of 2^e words (f may not overlap g): the product kernels on
// one transform of length 2^e for kMinLog <= e <= kMaxLog, otherwise
// natural-order transforms around a pointwise product (cyclic_mul_compose,
// which needs 16-byte aligned arrays when e >= 6).
int cyclic_mul_dev(u32* f, const u32* g, int e, u32 p, cudaStream_t st);
int cyclic_mul_compose(u32* f, const u32* g, int e, u32 p, cudaStream_t st);

}  // namespace cmb
