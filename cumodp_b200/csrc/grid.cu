// Bivariate products on the three-pass kernels (grid_product.cuh).
#include "grid_product.cuh"

#include <cstring>
#include <initializer_list>

#include "product.cuh"

namespace cmb {

namespace {

template <int E, int L2>
constexpr size_t grid_smem() {
    return (size_t)sizeof(u32) << grid_log(E, L2);
}

template <int E, int L2>
int launch_rows_t(const GridArgs& a, long long words, int dev, cudaStream_t st) {
    constexpr int LT = grid_log(E, L2);
    static DeviceOnce once;
    const int err = once(dev, [] {
        const cudaError_t e = allow_smem(k_grid_fwd_g<E, L2>, grid_smem<E, L2>());
        return e == cudaSuccess ? allow_smem(k_grid_mul_f<E, L2>, grid_smem<E, L2>()) : e;
    });
    if (err != OK) return err;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(words >> LT));
    cfg.blockDim = dim3(grid_threads(LT));
    cfg.dynamicSmemBytes = grid_smem<E, L2>();
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaEvent_t e0;
    bool tr = pass_timing_begin(st, &e0);
    cudaLaunchKernelEx(&cfg, k_grid_fwd_g<E, L2>, a);
    if (tr) pass_timing_end(st, "grid_fwd_g", e0);
    tr = pass_timing_begin(st, &e0);
    cudaLaunchKernelEx(&cfg, k_grid_mul_f<E, L2>, a);
    if (tr) pass_timing_end(st, "grid_mul_f", e0);
    return OK;
}

typedef int (*RowsFn)(const GridArgs&, long long, int, cudaStream_t);
const RowsFn kRows[3][kMaxRowLog + 1] = {
    {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, launch_rows_t<0, 6>, launch_rows_t<0, 7>, launch_rows_t<0, 8>,
     launch_rows_t<0, 9>, launch_rows_t<0, 10>, launch_rows_t<0, 11>, launch_rows_t<0, 12>, launch_rows_t<0, 13>,
     launch_rows_t<0, 14>},
    {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, launch_rows_t<1, 6>, launch_rows_t<1, 7>, launch_rows_t<1, 8>,
     launch_rows_t<1, 9>, launch_rows_t<1, 10>, launch_rows_t<1, 11>, launch_rows_t<1, 12>, launch_rows_t<1, 13>, nullptr},
    {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, launch_rows_t<2, 6>, launch_rows_t<2, 7>, launch_rows_t<2, 8>,
     launch_rows_t<2, 9>, launch_rows_t<2, 10>, launch_rows_t<2, 11>, launch_rows_t<2, 12>, nullptr, nullptr}};

}  // namespace

bool grid_split(int em, int en, int* l1, int* e) {
    if (em < 1 || en < kMinRowLog || em + en < 11) return false;
    // columns of 2^10 rows (the register kernels) first, then of 2^11
    for (const int c : {(int)kDefaultColLog, (int)kMaxColLog}) {
        *e = em > c ? em - c : 0;
        *l1 = em - *e;
        if (*e <= 2 && *e + en <= kMaxRowLog) return true;
    }
    return false;
}

int grid_mul_dev(u32* F, u32* G, int em, int en, u32 p, cudaStream_t st) {
    int err = OK, l1, E;
    if (!grid_split(em, en, &l1, &E)) return ASSUMPTION_ERROR;
    const PrimeCtx* pc = prime_ctx(p, &err);
    if (!pc) return err;
    const int dev = current_device(), l2 = E + en;
    const long long words = 1ll << (em + en);
    if ((err = ensure_kernel_attrs(dev)) != OK) return err;
    const Workspace ws_space(dev, kWsBiv, (size_t)2 * words * sizeof(u32), st, &err);
    u32* ws = ws_space.get();
    if (!ws) return err;
    const u32 wm = canonical_root(*pc, em), wn = canonical_root(*pc, en), wc = canonical_root(*pc, l1);
    const u32 ninv = powmod_exact((u32)(words % p), p - 2, p), scale = mulmod_exact(ninv, pc->info.r1, p);
    LargeArgs C;
    memset(&C, 0, sizeof(C));
    C.pk = C.pkc = make_prime_k_for(pc->info, wc, l1);
    C.twc = col_tables(dev, p, wc, l1, &err);
    GridArgs A;
    memset(&A, 0, sizeof(A));
    A.twr = row_tables(dev, p, wn, en, &err);
    if (!C.twc || !A.twr) return err;
    C.twc_inv = plan_tw_entries(col_plan(l1), l1);
    C.l1 = l1;
    C.l2 = l2;
    C.colpl = col_plan(l1);
    C.njobs = 1;
    A.pk = pc->pk;
    A.twr_inv = plan_tw_entries(row_plan(en), en);
    A.slots = 1 << l1;
    A.scale = tw_of(scale, p);
    A.wa = ws;
    A.wb = ws + words;
    if (E > 0 && !(A.lead = grid_lead_tables(dev, p, wm, em, en, l1, scale, &err))) return err;
    C.job0 = LargeJob{F, G, F, (int)words, (int)words, (int)words, 0, A.wa, A.wb};
    launch_col_fwd(C, 1, st);
    if ((err = kRows[E][en](A, words, dev, st)) != OK) return err;
    launch_col_inv(C, 1, st);
    return cuda_err(cudaGetLastError());
}

}  // namespace cmb
