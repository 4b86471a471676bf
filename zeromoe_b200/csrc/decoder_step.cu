// decoder_step.cu -- layer table and launch of the one-kernel decoder step.
#include <new>
#include <vector>

#include "zmoe_internal.h"

#include "decoder_step.cuh"

namespace zmoe {

using StepFn = void (*)(const StepArgs);

template <int GU, SmallSums SUMS>
static StepFn step_down(int dn) {
    switch (dn) {
    case Q2_K: return decoder_step_kernel<GU, Q2_K, SUMS>;
    case Q3_K: return decoder_step_kernel<GU, Q3_K, SUMS>;
    case Q4_K: return decoder_step_kernel<GU, Q4_K, SUMS>;
    }
    return nullptr;
}
template <SmallSums SUMS>
static StepFn pick_step(int gu, int dn) {
    switch (gu) {
    case Q2_K: return step_down<Q2_K, SUMS>(dn);
    case Q3_K: return step_down<Q3_K, SUMS>(dn);
    case Q4_K: return step_down<Q4_K, SUMS>(dn);
    }
    return nullptr;
}
static StepFn pick_sums(SmallSums sums, int gu, int dn) {
    return sums == SUMS_SHORT ? pick_step<SUMS_SHORT>(gu, dn) : sums == SUMS_LONG ? pick_step<SUMS_LONG>(gu, dn) : pick_step<SUMS_BLOCKS>(gu, dn);
}

struct DecoderStep {
    StepArgs a = {};
    StepFn fn = nullptr;
    size_t smem = 0;
    int n_sm = 0;
    StepLayer *table = nullptr;
    std::vector<zmoe_layer *> leaving;    // the last layer of each context
};

// [0, 1] grid barrier, [2, 3] arg-max key, then a ticket per KV head
int decoder_step_sync_words(int KV) { return 4 + KV; }

// The kernel's static arrays (1920 bytes), rounded up.  With more of them the request for all of STEP_SMEM fails when a decoder is created, and its
// steps are separate launches.
constexpr int STEP_STATIC = 2 * 1024, STEP_SMEM = 227 * 1024 - STEP_STATIC;

DecoderStep *decoder_step_create(const DecoderStepDesc &d) {
    int dev = 0, coop = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) return nullptr;
    const int QO = d.H * d.HD, G = d.H / d.KV, widest = d.D > QO ? d.D : QO;
    if (d.D % 256 || QO % 32 || d.D > 8192 || QO > 16384 || (reinterpret_cast<size_t>(d.head) & 15)) return nullptr;
    std::vector<StepLayer> table;
    std::vector<zmoe_layer *> leaving;
    int gu = -1, dn = -1, F = 0, E = 0, K = 0;
    for (int l = 0; l < d.n_layers; ++l) {
        if ((reinterpret_cast<size_t>(d.wqkv[l]) & 15) || (reinterpret_cast<size_t>(d.wo[l]) & 15)) return nullptr;
        RouterArgs r;
        SmallLaunch s;
        if (!layer_small_args(d.moe[l], d.xn, d.h, 1, 1, &r, &s) || r.D != d.D) return nullptr;
        if (l == 0) { gu = s.type_gu; dn = s.type_dn; F = s.F; E = r.E; K = r.K; }
        if (s.type_gu != gu || s.type_dn != dn || s.F != F || r.E != E || r.K != K) return nullptr;
        StepLayer L = {};
        L.attn_norm = d.attn_norm[l]; L.ffn_norm = d.ffn_norm[l];
        L.wqkv = static_cast<const uint8_t *>(d.wqkv[l]); L.wo = static_cast<const uint8_t *>(d.wo[l]);
        L.moe = small_args(r, s);
        L.leave_state = 1;
        for (int k = l + 1; k < d.n_layers; ++k)
            if (layer_context(d.moe[k]) == layer_context(d.moe[l])) L.leave_state = 0;
        if (L.leave_state) leaving.push_back(d.moe[l]);
        table.push_back(L);
    }
    if (table.empty()) return nullptr;
    // shared memory: what every CTA keeps, and as many rows on their way per warp as the rest has room for
    auto room = [](int bytes) { return (bytes + 47) & ~15; };
    const int rbd = d.D / 32 * 34, rbo = QO / 32 * 34;
    // from x on: a chunk of keys and values while attention runs
    const size_t from_x = (size_t)d.D * 4 + q8row_stride(d.D) + (size_t)K * q8row_stride(F) + ((size_t)2 * E + 8) * 4, kv = step_kv_bytes(d.HD);
    const size_t rest = widest + (size_t)((widest / 32 + 3) & ~3) * 4 + (size_t)G * d.HD * 4 + (from_x > kv ? from_x : kv);
    if (rest >= (size_t)STEP_SMEM) return nullptr;
    const int per_warp = (int)(((size_t)STEP_SMEM - rest) / SMALL_WARPS) & ~15;
    auto depth = [&](int bytes, int most) { const int n = per_warp / bytes; return n < most ? n : most; };
    const int q = room(rbd), o = room(rbo), g = 2 * room(table[0].moe.rb_gu), w = K * room(table[0].moe.rb_dn);
    const int nq = depth(q, 4), no = depth(o, 2), ng = depth(g, 4), nw = depth(w, 2);
    if (nq < 1 || no < 1 || ng < 1 || nw < 1) return nullptr;
    int stage = nq * q;
    for (int b : {no * o, ng * g, nw * w}) stage = b > stage ? b : stage;
    DecoderStep *s = new (std::nothrow) DecoderStep();
    if (!s) return nullptr;
    for (StepLayer &L : table) { L.moe.depth_gu = ng; L.moe.depth_dn = nw; L.moe.stage = stage; }
    s->fn = pick_sums(small_sums(1, K, d.D, F), gu, dn);
    s->smem = (size_t)SMALL_WARPS * stage + rest;
    s->n_sm = device_sm_count();
    s->leaving = leaving;
    if (!s->fn || s->n_sm <= 0 || raise_dynamic_smem(reinterpret_cast<const void *>(s->fn), STEP_SMEM) != ZMOE_OK ||
        cudaMalloc(reinterpret_cast<void **>(&s->table), table.size() * sizeof(StepLayer)) != cudaSuccess ||
        cudaMemcpy(s->table, table.data(), table.size() * sizeof(StepLayer), cudaMemcpyHostToDevice) != cudaSuccess) {
        decoder_step_destroy(s);
        return nullptr;
    }
    StepArgs &a = s->a;
    a.layers = s->table; a.n_layers = d.n_layers;
    a.embd = static_cast<const uint8_t *>(d.embd); a.head = static_cast<const uint8_t *>(d.head); a.out_norm = d.out_norm;
    a.D = d.D; a.H = d.H; a.KV = d.KV; a.HD = d.HD; a.vocab = d.vocab; a.max_ctx = d.max_ctx;
    a.eps = d.eps; a.theta_scale = d.theta_scale; a.scale = d.scale;
    a.h = d.h; a.xn = d.xn; a.qkv = d.qkv; a.part = d.part; a.logits = d.logits; a.aq = d.aq; a.ad = d.ad;
    a.kc = static_cast<__half *>(d.kc); a.vc = static_cast<__half *>(d.vc);
    a.pos = d.pos; a.next = d.next;
    a.bar = d.sync;
    a.best = reinterpret_cast<unsigned long long *>(d.sync + 2);
    a.head_ticket = d.sync + 4;
    a.splits = d.splits;
    a.stage = stage; a.depth_q = nq; a.depth_o = no;
    return s;
}

void decoder_step_destroy(DecoderStep *s) {
    if (!s) return;
    cudaFree(s->table);
    delete s;
}

int decoder_step_launch(DecoderStep *s, const int32_t *token_dev, cudaStream_t st) {
    for (zmoe_layer *L : s->leaving)
        if (context_path(layer_context(L)) >= 2) return ZMOE_ERR_STATE;
    StepArgs a = s->a;
    a.token = token_dev;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)s->n_sm);
    cfg.blockDim = dim3(SMALL_THREADS);
    cfg.dynamicSmemBytes = s->smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int rc = cooperative_status(cudaLaunchKernelEx(&cfg, s->fn, a));
    if (rc) return rc;
    count_launches(1);
    for (zmoe_layer *L : s->leaving) layer_small_done(L, a.xn, 1);
    return ZMOE_OK;
}

}  // namespace zmoe
