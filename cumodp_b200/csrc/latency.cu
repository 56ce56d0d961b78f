// Host side of the one-launch products (latency_product.cuh).
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "product.cuh"

namespace cmb {

namespace {

constexpr int kMaxOneCtaLog = 11;  // longest transform of the single-CTA form

template <int LOGL, int CL, int NP, bool WIDE>
cudaError_t launch_t(const LatArgs<NP>& a, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CL, NP);
    cfg.blockDim = dim3(lat_threads(LOGL));
    cfg.dynamicSmemBytes = lat_smem(LOGL, CL);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = CL > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k_latency_product<LOGL, CL, NP, WIDE>, a);
}

// Sets the kernel's limits on the current device; whether it can run there.
template <int LOGL, int CL, int NP, bool WIDE>
bool setup_np() {
    const void* f = (const void*)k_latency_product<LOGL, CL, NP, WIDE>;
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lat_smem(LOGL, CL)) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (CL == 1) return true;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CL);
    cfg.blockDim = dim3(lat_threads(LOGL));
    cfg.dynamicSmemBytes = lat_smem(LOGL, CL);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int fit = 0;
    if (cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&fit, f, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return fit > 0;
}

template <int LOGL, int CL>
bool setup_t() {
    return setup_np<LOGL, CL, 1, false>() && setup_np<LOGL, CL, 3, false>() && setup_np<LOGL, CL, 2, true>() &&
           setup_np<LOGL, CL, 3, true>();
}

struct Form {
    int logl;
    cudaError_t (*one)(const LatArgs<1>&, cudaStream_t);
    cudaError_t (*three)(const LatArgs<3>&, cudaStream_t);
    cudaError_t (*wide2)(const LatArgs<2>&, cudaStream_t);
    cudaError_t (*wide3)(const LatArgs<3>&, cudaStream_t);
    bool (*setup)();
};
template <int LOGL, int CL>
constexpr Form form() {
    return Form{LOGL,
                launch_t<LOGL, CL, 1, false>,
                launch_t<LOGL, CL, 3, false>,
                launch_t<LOGL, CL, 2, true>,
                launch_t<LOGL, CL, 3, true>,
                setup_t<LOGL, CL>};
}
// by log2 of the transform length, from kMinLog on
const Form kForms[] = {form<5, 1>(),  form<6, 1>(),  form<7, 1>(),  form<8, 1>(),   form<9, 1>(),   form<10, 1>(),
                       form<11, 1>(), form<8, 16>(), form<9, 16>(), form<10, 16>(), form<11, 16>(), form<12, 16>()};
static_assert(sizeof(kForms) / sizeof(kForms[0]) == kMaxLatencyLog - kMinLog + 1, "one form per length");
static_assert(kMaxOneCtaLog - kMinLog + 1 == 7, "the single-CTA forms come first");

// A prime's part of a launch, kept per device, prime and length beside the
// tables it points to (a product's constants take a dozen modular powers on
// the host); `usable` = false where the kernels cannot run.
struct Prepared {
    LatPrime pr;
    bool usable;
};

const char* const kName[] = {"latency_product_5",  "latency_product_6",  "latency_product_7",  "latency_product_8",
                             "latency_product_9",  "latency_product_10", "latency_product_11", "latency_product_12",
                             "latency_product_13", "latency_product_14", "latency_product_15", "latency_product_16"};

int prepared(const PrimeCtx& pc, int logn, int dev, Prepared* out) {
    static std::mutex m;
    static std::map<std::tuple<int, u32, int>, Prepared>* cache = new std::map<std::tuple<int, u32, int>, Prepared>();
    const Form& form = kForms[logn - kMinLog];
    std::lock_guard<std::mutex> g(m);
    const auto key = std::make_tuple(dev, pc.info.p, logn);
    auto it = cache->find(key);
    if (it == cache->end()) {
        Prepared n{};
        n.usable = form.setup();
        if (n.usable) {
            const u32 p = pc.info.p, root = canonical_root(pc, logn);
            int err = OK;
            const Tw* t = latency_tables(dev, p, root, logn, form.logl, &err);
            if (!t) return err;
            const u32 ninv = powmod_exact((u32)((1ull << logn) % p), p - 2, p);
            n.pr.pk = pc.pk;
            n.pr.scale = tw_of(mulmod_exact(ninv, pc.info.r1, p), p);
            n.pr.r32 = tw_of(pc.info.r1, p);
            n.pr.tw = t;
            n.pr.lead = t + 2 * lat_entries(form.logl);
        }
        it = cache->emplace(key, n).first;
    }
    *out = it->second;
    return OK;
}

}  // namespace

namespace {

// The library code of a launch; one that was refused for resources (the room
// the set-up found for a cluster is gone) leaves *launched false and no error,
// and the caller takes the other kernels.
int launch_result(cudaError_t e, bool* launched) {
    *launched = e == cudaSuccess;
    if (e == cudaErrorLaunchOutOfResources || e == cudaErrorInvalidClusterSize) {
        cudaGetLastError();
        return OK;
    }
    return cuda_err(e);
}

}  // namespace

int latency_usable(const PrimeCtx& pc, int logn, int dev, bool* usable) {
    Prepared P{};
    const int err = prepared(pc, logn, dev, &P);
    *usable = err == OK && P.usable;
    return err;
}

int latency_mul(const PrimeCtx& pc, int logn, int dev, const ProdJob& job, cudaStream_t st, bool* launched) {
    *launched = false;
    Prepared P;
    const int err = prepared(pc, logn, dev, &P);
    if (err != OK || !P.usable) return err;
    const LatArgs<1> a{{P.pr}, job.a, job.b, job.h, job.la, job.lb, job.lh, 0, 0, 0};
    NvtxRange range(kName[logn - kMinLog]);
    cudaEvent_t e0;
    const bool tr = pass_timing_begin(st, &e0);
    const cudaError_t ce = kForms[logn - kMinLog].one(a, st);
    if (tr) pass_timing_end(st, kName[logn - kMinLog], e0);
    return launch_result(ce, launched);
}

namespace {

int prepared_all(const u32* primes, int np, int logn, int dev, Prepared* P, bool* usable) {
    *usable = false;
    for (int r = 0; r < np; ++r) {
        int err = OK;
        const PrimeCtx* pc = prime_ctx(primes[r], &err);
        if (!pc) return err;
        if (logn > pc->info.two_adic) return FFT_SIZE_TOO_LARGE;
        if ((err = prepared(*pc, logn, dev, &P[r])) != OK) return err;
        if (!P[r].usable) return OK;
    }
    *usable = true;
    return OK;
}

}  // namespace

int latency_mul_primes(const u32* primes, int np, int dev, const u32* a, int la, long long astride, const u32* b, int lb,
                       long long bstride, u32* h, long long hstride, cudaStream_t st, bool* launched) {
    *launched = false;
    const int logn = product_logn(la, lb), lh = la + lb - 1;
    if (np < 3 || np > 4 || logn > kMaxLatencyLog) return OK;
    Prepared P[4];
    bool usable;
    const int err = prepared_all(primes, np, logn, dev, P, &usable);
    if (err != OK || !usable) return err;
    const Form& form = kForms[logn - kMinLog];
    cudaEvent_t e0;
    const bool tr = pass_timing_begin(st, &e0);
    cudaError_t ce =
        form.three(LatArgs<3>{{P[0].pr, P[1].pr, P[2].pr}, a, b, h, la, lb, lh, astride, bstride, hstride}, st);
    if (np == 4 && ce == cudaSuccess)
        ce = form.one(LatArgs<1>{{P[3].pr}, a + 3 * astride, b + 3 * bstride, h + 3 * hstride, la, lb, lh, 0, 0, 0}, st);
    if (tr) pass_timing_end(st, kName[logn - kMinLog], e0);
    return launch_result(ce, launched);
}

int latency_mul_i64(const u32* primes, int np, int dev, const long long* a, int la, const long long* b, int lb, u32* h,
                    cudaStream_t st, bool* launched) {
    *launched = false;
    const int logn = product_logn(la, lb), lh = la + lb - 1;
    if (np < 2 || np > 3 || logn > kMaxLatencyLog) return OK;
    Prepared P[3];
    bool usable;
    const int err = prepared_all(primes, np, logn, dev, P, &usable);
    if (err != OK || !usable) return err;
    const Form& form = kForms[logn - kMinLog];
    cudaEvent_t e0;
    const bool tr = pass_timing_begin(st, &e0);
    const cudaError_t ce =
        np == 2 ? form.wide2(LatArgs<2>{{P[0].pr, P[1].pr}, a, b, h, la, lb, lh, 0, 0, lh}, st)
                : form.wide3(LatArgs<3>{{P[0].pr, P[1].pr, P[2].pr}, a, b, h, la, lb, lh, 0, 0, lh}, st);
    if (tr) pass_timing_end(st, kName[logn - kMinLog], e0);
    return launch_result(ce, launched);
}

namespace {

template <int LOGL>
int launch_level_t(const LevelArgs& a, int dev, cudaStream_t st) {
    constexpr size_t smem = lat_smem(LOGL, 1);
    static DeviceOnce once;
    const int err = once(dev, [] { return allow_smem(k_monic_level<LOGL>, smem); });
    if (err != OK) return err;
    const int grid = std::min(a.npairs, sm_count(dev) * level_ctas(LOGL));
    k_monic_level<LOGL><<<grid, level_threads(LOGL), smem, st>>>(a);
    return cuda_err(cudaGetLastError());
}
typedef int (*LevelFn)(const LevelArgs&, int, cudaStream_t);
const LevelFn kLevel[] = {launch_level_t<5>, launch_level_t<6>,  launch_level_t<7>,  launch_level_t<8>,
                          launch_level_t<9>, launch_level_t<10>, launch_level_t<11>, launch_level_t<12>};

}  // namespace

int monic_level_dev(const PrimeCtx& pc, int l, int npairs, const u32* in, u32* out, cudaStream_t st) {
    int logn = kMinLog, err = OK;
    while ((1 << logn) < 2 * l) ++logn;
    if (logn > kMaxLevelLog) return ASSUMPTION_ERROR;
    if (logn > pc.info.two_adic) return FFT_SIZE_TOO_LARGE;
    const int dev = current_device();
    const u32 p = pc.info.p, root = canonical_root(pc, logn);
    LevelArgs a{};
    // these lengths' block tables are those of the one-launch product where it
    // has one CTA; 2^12 has a table of its own
    a.pr.tw = latency_tables(dev, p, root, logn, logn, &err);
    if (!a.pr.tw) return err;
    const u32 ninv = powmod_exact((u32)((1ull << logn) % p), p - 2, p);
    a.pr.pk = pc.pk;
    a.pr.scale = tw_of(mulmod_exact(ninv, pc.info.r1, p), p);
    a.in = in;
    a.out = out;
    a.l = l;
    a.npairs = npairs;
    cudaEvent_t e0;
    const bool tr = pass_timing_begin(st, &e0);
    err = kLevel[logn - kMinLog](a, dev, st);
    if (tr) pass_timing_end(st, "monic_level", e0);
    return err;
}

}  // namespace cmb
