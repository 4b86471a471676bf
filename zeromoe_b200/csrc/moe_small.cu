// moe_small.cu -- launch of the one-kernel MoE layer for calls of very few pairs.
#include "moe_small.cuh"
#include "zmoe_internal.h"

namespace zmoe {

using SmallFn = void (*)(const SmallArgs);

template <int GU, SmallSums SUMS>
static SmallFn pick_down(int dn) {
    switch (dn) {
    case Q2_K: return moe_small_kernel<GU, Q2_K, SUMS>;
    case Q3_K: return moe_small_kernel<GU, Q3_K, SUMS>;
    case Q4_K: return moe_small_kernel<GU, Q4_K, SUMS>;
    }
    return nullptr;
}
template <SmallSums SUMS>
static SmallFn pick_small(int gu, int dn) {
    switch (gu) {
    case Q2_K: return pick_down<Q2_K, SUMS>(dn);
    case Q3_K: return pick_down<Q3_K, SUMS>(dn);
    case Q4_K: return pick_down<Q4_K, SUMS>(dn);
    }
    return nullptr;
}
static SmallFn pick_sums(SmallSums sums, int gu, int dn) {
    return sums == SUMS_SHORT ? pick_small<SUMS_SHORT>(gu, dn) : sums == SUMS_LONG ? pick_small<SUMS_LONG>(gu, dn) : pick_small<SUMS_BLOCKS>(gu, dn);
}

// shared memory of the kernel's static arrays (896 bytes), rounded up; a launch asks for all of SMALL_SMEM, so a build with more of them is refused
constexpr int SMALL_STATIC = 1024, SMALL_SMEM = 227 * 1024 - SMALL_STATIC;

// Rows on their way per warp and the bytes they take; 0 where a shape does not fit
static size_t small_geometry(int gu, int dn, int T, int D, int F, int E, int K, int *depth_gu, int *depth_dn, int *stage) {
    const int room_gu = ((D / QK_K) * block_bytes(gu) + 47) & ~15, room_dn = ((F / QK_K) * block_bytes(dn) + 47) & ~15;
    const size_t rest = (size_t)T * q8row_stride(D) + (size_t)T * K * q8row_stride(F) + ((size_t)2 * E * T + 8) * sizeof(float);
    if (rest >= (size_t)SMALL_SMEM) return 0;
    const int per_warp = (int)(((size_t)SMALL_SMEM - rest) / SMALL_WARPS) & ~15;
    int dg = per_warp / (2 * room_gu), dd = per_warp / (K * room_dn);
    if (dg < 1 || dd < 1) return 0;
    if (dg > 4) dg = 4;
    if (dd > 2) dd = 2;
    const int sg = dg * 2 * room_gu, sd = dd * K * room_dn;
    *depth_gu = dg; *depth_dn = dd; *stage = sg > sd ? sg : sd;
    return (size_t)SMALL_WARPS * *stage + rest;
}

bool moe_small_supported(int gu, int dn, int T, int D, int F, int E, int K) {
    int a, b, c;
    return T >= 1 && T <= SMALL_WARPS && (long)T * K <= SMALL_PAIRS && K <= SMALL_PAIRS && D % QK_K == 0 && F % QK_K == 0 && D <= 8192 && F <= 8192 &&
           small_geometry(gu, dn, T, D, F, E, K, &a, &b, &c) != 0;
}

SmallArgs small_args(const RouterArgs &r, const SmallLaunch &L) {
    SmallArgs a = {};
    a.x = r.x; a.wr = r.wr; a.bias = r.bias;
    a.T = r.T; a.D = r.D; a.F = L.F; a.E = r.E; a.K = r.K;
    a.sp = RouterSpec{r.E, r.K, r.gating, r.normalize, r.weight_scale, r.n_groups, r.n_groups_used};
    a.wg = static_cast<const uint8_t *>(L.w_gate); a.wu = static_cast<const uint8_t *>(L.w_up); a.wd = static_cast<const uint8_t *>(L.w_down);
    a.sg = L.stride_gate; a.su = L.stride_up; a.sd = L.stride_down;
    a.rb_gu = (r.D / QK_K) * block_bytes(L.type_gu);
    a.rb_dn = (L.F / QK_K) * block_bytes(L.type_dn);
    a.clamp = L.clamp; a.clamp_fused = L.clamp_fused;
    a.logits = r.logits; a.ids = r.ids; a.weights = r.weights; a.q8x = r.q8x;
    a.act = L.act; a.out = L.out; a.accumulate = L.accumulate;
    a.plan = PlanOut{r.plan.hdr, r.plan.active, r.plan.offs, r.plan.slot, r.plan.item_offs_gu, r.plan.item_offs_dn, r.plan.freq, r.plan.aoffs,
                     r.plan.antok, r.nrt_gu, r.nrt_dn, r.plan.pos, r.plan.mt_gu, r.plan.mt_dn};
    a.err = L.err; a.bad = L.bad; a.bar = L.bar;
    return a;
}

int launch_moe_small(const RouterArgs &r, const SmallLaunch &L, cudaStream_t st) {
    SmallArgs a = small_args(r, L);
    const size_t smem = small_geometry(L.type_gu, L.type_dn, r.T, r.D, L.F, r.E, r.K, &a.depth_gu, &a.depth_dn, &a.stage);
    SmallFn fn = pick_sums(small_sums(r.T, r.K, r.D, L.F), L.type_gu, L.type_dn);
    if (!smem || !fn) return ZMOE_ERR_SHAPE;
    if (raise_dynamic_smem(reinterpret_cast<const void *>(fn), SMALL_SMEM) != ZMOE_OK) return ZMOE_ERR_CUDA;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)r.n_sm);
    cfg.blockDim = dim3(SMALL_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cooperative_status(cudaLaunchKernelEx(&cfg, fn, a));
}

}  // namespace zmoe
