// api.cu -- the C ABI of libzmoe_b200.so (declared in include/zmoe_b200.h):
// reference kernel-launch symbols, the ggml-style op hook on plain tensor
// mirrors, and the layer-level entry with its per-device context.
#include <atomic>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <utility>

#include "zmoe_common.cuh"
#include "zmoe_internal.h"

using namespace zmoe;

namespace {

std::atomic<uint64_t> g_launches{0};
std::atomic<uint64_t> g_hook_launches{0};
thread_local int tl_status = ZMOE_OK;

inline int ok(cudaError_t e) { return e == cudaSuccess ? ZMOE_OK : ZMOE_ERR_CUDA; }

template <typename T>
int dev_alloc(T **p, size_t n) {
    *p = nullptr;
    if (n == 0) n = 1;
    return ok(cudaMalloc(reinterpret_cast<void **>(p), n * sizeof(T)));
}

int sm_count() { return zmoe::device_sm_count(); }

// pairs per expert, averaged over the call, from which the layer entry takes the tensor-core grouped GEMM
constexpr int kGemmMinPairsPerExpert = 24;

struct PlanStore {
    PlanBuffers b;
    int cap_e = 0, cap_p = 0;
    int alloc(int E, int P) {
        int rc = 0;
        rc |= dev_alloc(&b.hdr, 4);
        rc |= dev_alloc(&b.active, E);
        rc |= dev_alloc(&b.offs, E + 1);
        rc |= dev_alloc(&b.slot, P);
        rc |= dev_alloc(&b.item_offs_gu, E + 1);
        rc |= dev_alloc(&b.item_offs_dn, E + 1);
        rc |= dev_alloc(&b.freq, E);
        rc |= dev_alloc(&b.aoffs, E);
        rc |= dev_alloc(&b.antok, E);
        rc |= dev_alloc(&b.pos, P);
        b.cap_e = E;
        cap_e = E;
        cap_p = P;
        return rc ? ZMOE_ERR_CUDA : ZMOE_OK;
    }
    void release() {
        cudaFree(b.hdr); cudaFree(b.active); cudaFree(b.offs); cudaFree(b.slot);
        cudaFree(b.item_offs_gu); cudaFree(b.item_offs_dn); cudaFree(b.freq); cudaFree(b.aoffs); cudaFree(b.antok); cudaFree(b.pos);
        b = PlanBuffers();
        cap_e = cap_p = 0;
    }
};

}  // namespace

namespace zmoe {

int device_sm_count() {
    constexpr int kMax = 64;
    static std::atomic<int> cache[kMax];
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (dev >= 0 && dev < kMax && (n = cache[dev].load(std::memory_order_relaxed)) > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (dev >= 0 && dev < kMax) cache[dev].store(n, std::memory_order_relaxed);
    return n;
}

void count_launches(uint64_t n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
void set_last_status(int rc) { tl_status = rc; }

int raise_dynamic_smem(const void *fn, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, size_t> done;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return ZMOE_ERR_CUDA;
    std::lock_guard<std::mutex> lock(mu);
    size_t &have = done[std::make_pair(fn, dev)];
    if (have < bytes) {
        if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
            return ZMOE_ERR_CUDA;
        have = bytes;
    }
    return ZMOE_OK;
}

}  // namespace zmoe

// ---------------------------------------------------------------------------
// context and layer
// ---------------------------------------------------------------------------
// Decode kernels of the two projections of a call (see zmoe_layer), the item spaces of a plan for them, and the layouts of the
// quantised rows they read
enum KernelSet { SET_SMALL, SET_BIG, SET_TC };
struct CallGeom {
    KernelSet gu = SET_SMALL, dn = SET_SMALL;
    int mt_gu = 0, mt_dn = 0, nrt_gu = 0, nrt_dn = 0;   // pairs per item, row tiles per expert
    int experts = 0, topk = 0, layout_gate = 0, layout_up = 0;
    bool operator==(const CallGeom &o) const {
        return gu == o.gu && dn == o.dn && mt_gu == o.mt_gu && mt_dn == o.mt_dn && nrt_gu == o.nrt_gu && nrt_dn == o.nrt_dn && experts == o.experts &&
               topk == o.topk && layout_gate == o.layout_gate && layout_up == o.layout_up;
    }
};

struct zmoe_ctx {
    int max_t = 0, max_d = 0, max_f = 0, max_e = 0, max_k = 0;
    int n_sm = 0;
    int device = 0;
    uint8_t *q8x = nullptr;    // packed Q8_K rows of the layer input (unit layout of the gate format)
    uint8_t *q8x2 = nullptr;   // the same in the other unit layout, for an up format that needs it
    float *act = nullptr;      // [P, F] SwiGLU output
    float *act2 = nullptr;     // [2, P, F] gate / up when their types differ (lazy)
    uint8_t *q8act = nullptr;  // packed Q8_K rows of act
    void *xq_f16 = nullptr;   // [P, D] fp16: layer input rows in expert order after the Q8_K round trip
    void *actq_f16 = nullptr; // [P, F] fp16: act after the Q8_K round trip (tensor-core path)
    float *xscale = nullptr, *actscale = nullptr;  // per-row powers of two of the fp16 copies
    int32_t *zero_ids = nullptr;   // [T] zeros / ones: routes of a dense (single-expert) FFN
    float *one_w = nullptr;
    float *gate_s = nullptr;       // [T] per-token scalar gates of a gated shared expert
    const float *x_last = nullptr;  // the activations the current route table was built from
    int path = 0;              // 0 auto, 1 decode kernels, 2 tensor-core GEMM, 3 decode kernels, scalar path only
    float *ydown = nullptr;    // [P, D] per-pair down-projection output
    float *logits = nullptr;   // [T, E] router logits, then probabilities
    float *logits_part = nullptr;  // [router_part_rows, E] partial logits of the tiled router (contexts of > ROUTER_TILED_TOKENS tokens)
    bool q8x_valid = false;    // q8x (and q8x2) hold the quantised rows of x_last
    int32_t *ids = nullptr;    // [T, K]
    float *weights = nullptr;  // [T, K]
    PlanStore plan;
    int *err = nullptr;
    int *bad = nullptr;        // [2] NaN / Inf inputs seen by the fused SwiGLU epilogues
    int *queue = nullptr;      // [4] item tickets of the decode matmuls (two per projection; every launch leaves them zero)
    unsigned *ticket = nullptr;
    unsigned *small_bar = nullptr;  // [2] grid-barrier counters of the one-kernel layer (every launch leaves them zero)
    float *x_stage = nullptr, *out_stage = nullptr;  // device staging of the host entry
    cudaStream_t host_stream = nullptr;
    int *err_host = nullptr;   // pinned mirror of err: the host entry reads the flag with the same sync as its output
    int routed_t = -1;  // tokens of the current route table
    CallGeom planned;         // what the current plan and quantised rows were made for: set by the calls that make them, and by nothing else
};

struct zmoe_layer {
    zmoe_ctx *ctx;
    zmoe_layer_desc d;
    // Geometries, tile maps and item spaces of the decode kernels.  Three sets: `big` (the K-chunked kernel where
    // the shapes allow it), `small` (the kernel whose whole CTA works on one 16-row item: shorter latency
    // when there are fewer items than warp sets to give them to: calls of at most kSmallCallPairs pairs) and `tc` (integers on the tensor cores).  The plan of a call is
    // built for one of them per projection (call_geom).
    struct Proj {
        MmidGeom g_gu, g_gate1, g_dn;
        CUtensorMap tm_gate, tm_up, tm_down;
        bool has_tm_gu = false, has_tm_dn = false;
        int nrt_gu = 0, nrt_dn = 0;
        int mt_gu = 4, mt_dn = 4;   // pairs per item of the two projections
    } big, small, tc;
    const Proj &set(KernelSet s) const { return s == SET_SMALL ? small : s == SET_BIG ? big : tc; }
    bool dual;
    bool gemm_shape = false;    // the shapes allow the tensor-core grouped GEMM
    size_t bytes_gate, bytes_up, bytes_down;
    bool whole = true;          // these hold every row of every expert: the one-kernel forms read whole rows, the others stop at the end
};
// Layers whose calls of T tokens the one-kernel forms take: the pairs' experts hold at most this many bytes, and no IQ2_XXS, whose
// one-pair dot is bound by its table lookups.  One kernel saves about 10 us of launches and plans, and its rows come a little slower
// than those of the kernels it stands for.  us per layer, one kernel / five launches, by MiB: Q4_K 2048 / 768: two tokens (40) 28.8 / 37.8, three
// (61) 37.9 / 47.2, four (81) 50.0 / 51.1; 4096 / 1536, one token: Q2_K and Q3_K (52) 36.9 / 42.2, Q3_K (62) 41.3 / 48.8; two: Q2_K and
// Q3_K (105) 60.3 / 52.8.  The decoder step, us for four layers, one kernel / separate launches: 4096 / 1536, Q2_K and Q3_K (52) 327 / 366, Q3_K
// (62) 363 / 391, at position 1024 400 / 514; Q4_K 2048 / 768 (20) 207 / 284.
static const size_t kFusedCallBytes = (size_t)64 << 20;
static bool takes_fused(const zmoe_layer_desc &d, int T) {
    const size_t gu = (size_t)d.d_ff * (d.d_model / QK_K) * (block_bytes(d.gate.type) + block_bytes(d.up.type));
    const size_t dn = (size_t)d.d_model * (d.d_ff / QK_K) * block_bytes(d.down.type);
    if (d.n_experts > 256 || d.n_groups > 1) return false;             // what its router holds in registers
    return d.gate.type != IQ2_XXS && d.down.type != IQ2_XXS && (size_t)T * d.topk * (gu + dn) <= kFusedCallBytes;
}

// A layer call runs as one kernel only where what every CTA quantises for itself, the tokens' and the pairs' rows, is little too, counted in blocks
// of 256 (about 0.15 us for one).  us per layer, one kernel / five launches, experts chosen evenly | by a router with favourites (Zipf 1.1), whose
// shared rows the launches read once and the one kernel once per pair; "3 of 8": tokens of experts.
//   Up to 64 blocks, from 2048 output rows on: Q4_K 2048 / 768, 2 of 8 28.8 / 37.8 | 30.1 / 37.7, 4096 / 1024, 2 of 4 31.8 / 41.1 | 32.5 / 43.4, 7168 / 256, 2 of
//   2 27.7 / 27.5 | 27.9 / 28.3.  Fewer rows share that cost among less work: up to 48, Q4_K 1024 / 512, 4 of 4 22.3 / 29.5 | 22.5 / 27.1, 512 / 256, 8 of 4
//   23.3 / 30.4 | 23.4 / 32.2; above, 256 / 2048, 3 of 2 (51) 22.9 / 21.9, 512 / 8192, 1 of 2 (66) 25.4 / 23.4.
//   65 to 96, up to three tokens, to 80 with more: the launches' time grows with the pairs' rows on their way, so a token needs a few experts.  Q4_K 2048 /
//   768, 3 of 8 (96) 37.9 / 47.2 | 39.1 / 39.4, 4 of 4 (80) 31.1 / 35.6 | 31.5 / 33.5, 7168 / 256, 3 of 4 (96) 40.5 / 52.3 | 40.1 / 53.2, 8192 / 1024, 2 of 2 (80)
//   37.5 / 42.1 | 36.7 / 41.4; Q2_K 4096 / 512, 3 of 4 (72) 34.5 / 35.4 | 34.2 / 35.3; Q3_K 2048 / 1024, 3 of 4 (72) 20 and 13 % less.  Not taken: Q4_K 3072 / 768, 4
//   of 4 (96) 43.2 / 42.2 | 42.7 / 37.7, 2048 / 2048, 4 of 2 (96) 35.9 / 40.9 | 36.1 / 27.4, 7168 / 256, 3 of 2 (90) 34.9 / 32.3 | 34.5 / 32.0, 8192 / 2048,
//   2 of 1 (80) 41.9 / 40.1 | 41.1 / 38.4, 4096 / 1536, 4 of 1 (88) 38.5 / 35.9 | 38.2 / 29.3.
//   Of 178 shapes in that range (Q4_K, Q3_K, Q2_K with Q3_K; 2048 to 8192 / 256 to 3072; 1 to 8 tokens of 1 to 10 experts) the 97 taken are 11.7 %
//   faster on average as one kernel with evenly chosen experts, 7.6 % with favourites (worst: 11 and 14 % slower), the 81 not taken 0.3 and 12.0 % slower.
// Above 64 also only with twice as many experts as pairs or more, as in all of these: among fewer, evenly chosen experts are shared too (2048 / 768, 3 of 8
// of 32 experts 37.5 / 42.7 | 37.8 / 36.9).  (The decoder step saves far more launches and does not ask.)
static bool repeats_little(const zmoe_layer_desc &d, int T) {
    const long pairs = (long)T * d.topk, blocks = (long)T * (d.d_model / QK_K) + pairs * (d.d_ff / QK_K);
    if (blocks <= (d.d_model < 2048 ? 48 : 64)) return true;
    return blocks <= (T <= 3 ? 96 : 80) && d.topk >= (T <= 2 ? 2 : 3) && d.d_model >= 2048 && 2 * pairs <= d.n_experts;
}

namespace zmoe {
int layer_route_table(zmoe_layer *L, const int32_t **ids_dev, const float **weights_dev, int *n_experts) {
    if (!L || !ids_dev || !weights_dev || !n_experts) return ZMOE_ERR_ARG;
    if (L->ctx->routed_t <= 0) return ZMOE_ERR_STATE;
    *ids_dev = L->ctx->ids;
    *weights_dev = L->ctx->weights;
    *n_experts = L->d.n_experts;
    return ZMOE_OK;
}
zmoe_ctx *layer_context(zmoe_layer *L) { return L ? L->ctx : nullptr; }
int context_path(const zmoe_ctx *c) { return c ? c->path : 0; }
}  // namespace zmoe

// The kernel of one projection of a call of P pairs: the integer tensor-core kernel (mmid_tc.cuh) from so many pairs per expert on,
// on average, that its one conversion of a weight for up to 32 pairs pays; below, the kernels that convert it for up to eight (six, four) pairs
// and keep more of the machine busy with few.  `other` is their geometry, `nrt` the kernel's row tiles per expert, `dual` gate and up at once.
// A layer of 4096 / 1536, 128 experts, us, that kernel against those before it:
//   IQ2_XXS  8 tokens 209 / 241, 61 498 / 826, 256 594 / 2608; 2048 / 768: 8 tokens 82 / 99, 40 150 / 280, 200 187 / 1006
//   Q3_K     (no chunk geometry at 4096) 24 tokens 310 / 342, 61 410 / 585, 256 558 / 1916
//   Q2_K     gate and up 14 pairs per expert +19, 16 -1, 18 -14; down 14 -34
// One item takes its time however few there are, so few experts need more pairs: the second conditions.  They lie where the two meet
// with 1 to 16 experts, P against that kernel - those before it, us:
//   gate and up, rows of up to 16 super-blocks: IQ2_XXS 4096 / 1536 16 +2, 24 -4, 2048 / 768 32 +2, 48 -3, 4096 / 512 48 +2, 64 -1;
//     Q3_K 4096 / 1536 16 +5, 24 +2, 32 -5.  (Longer rows: 5120 / 1536 from 9 on, -6; rows the other kernel cannot share among pairs: from 9 on.)
//   down, against the chunk geometry: IQ2_XXS 4096 / 1536 16 +3, 32 -2, 48 -3, 2816 / 1024 48 +3, 80 -2; Q3_K 4096 / 1536 16 +2, 48 -3;
//     without one: Q3_K 2048 / 2048 16 +3, 32 -1, 48 -5
//   Q2_K: 32 experts, gate and up 576 +5, 704 -3 (7168 / 2048, 8 to 128 experts, 16 per expert -3 to -32); down 8 experts 112 -3, 4 experts
//     64 +2
// From 24 per expert on only calls that the grouped GEMM does not take come here.
static bool takes_tc(int type, int I, bool dual, int nrt, const MmidGeom &other, long P, int E) {
    const int nb = I / QK_K;
    if (type != IQ2_XXS && type != Q3_K && type != Q2_K) return false;
    if (P >= 24L * E) return true;
    if (type == Q2_K) return dual ? P >= (nb > 16 ? 16L : 18L) * E && (nb > 16 || P >= 1024) : P >= 14L * E && P >= 112;
    if (type == IQ2_XXS ? 2 * P < E : other.v2 ? P < 5L * E : 2 * P < 3L * E) return false;
    if (other.v2) return P * nrt * nb >= 7168;
    if (nb > 16 || !mmid_shares_rows(type, other, I, dual)) return true;
    return dual ? P * nrt >= 576 : P * nrt * nb >= 4096;
}

// g with all but the sets it names as this layer has it for T tokens
static CallGeom on_layer(const zmoe_layer *L, int T, CallGeom g) {
    const zmoe_layer::Proj &u = L->set(g.gu), &d = L->set(g.dn);
    g.mt_gu = g.gu == SET_TC ? tc_maxtok(T) : u.mt_gu;
    g.mt_dn = g.dn == SET_TC ? tc_maxtok(T) : d.mt_dn;
    g.nrt_gu = u.nrt_gu;
    g.nrt_dn = d.nrt_dn;
    g.experts = L->d.n_experts; g.topk = L->d.topk;
    g.layout_gate = q8_layout_of(L->d.gate.type); g.layout_up = q8_layout_of(L->d.up.type);
    return g;
}
// the kernels of a call of T tokens; path: what the context is set to
static CallGeom call_geom(const zmoe_layer *L, int T, int path) {
    const long P = (long)T * L->d.topk;
    const int E = L->d.n_experts;
    CallGeom g;
    g.gu = g.dn = P <= kSmallCallPairs ? SET_SMALL : SET_BIG;
    if (P > kSmallCallPairs && path != 3) {
        const int D = L->d.d_model, nrt = L->tc.nrt_gu;
        if (L->tc.has_tm_gu && takes_tc(L->d.gate.type, D, L->dual, nrt, L->big.g_gu, P, E) &&
            (L->dual || takes_tc(L->d.up.type, D, false, nrt, L->big.g_gate1, P, E)))
            g.gu = SET_TC;
        if (L->tc.has_tm_dn && takes_tc(L->d.down.type, L->d.d_ff, false, L->tc.nrt_dn, L->big.g_dn, P, E)) g.dn = SET_TC;
    }
    return on_layer(L, T, g);
}
// whether this layer's kernels can read a plan made for g: not where another layer of the context, of other shapes or formats, made it
static bool plan_fits(const zmoe_layer *L, int T, const CallGeom &g) {
    return (g.gu != SET_TC || L->tc.has_tm_gu) && (g.dn != SET_TC || L->tc.has_tm_dn) && on_layer(L, T, g) == g;
}

extern "C" {

int zmoe_ctx_create(int max_tokens, int max_d_model, int max_d_ff, int max_experts, int max_topk, zmoe_ctx **out) {
    if (!out || max_tokens <= 0 || max_d_model <= 0 || max_d_ff <= 0 || max_experts <= 0 || max_topk <= 0)
        return ZMOE_ERR_ARG;
    if (max_d_model % QK_K || max_d_ff % QK_K) return ZMOE_ERR_SHAPE;
    zmoe_ctx *c = new (std::nothrow) zmoe_ctx();
    if (!c) return ZMOE_ERR_ARG;
    c->max_t = max_tokens; c->max_d = max_d_model; c->max_f = max_d_ff; c->max_e = max_experts; c->max_k = max_topk;
    c->n_sm = sm_count();
    cudaGetDevice(&c->device);
    const size_t P = (size_t)max_tokens * max_topk;
    int rc = c->n_sm > 0 ? 0 : ZMOE_ERR_CUDA;
    rc |= dev_alloc(&c->q8x, (size_t)max_tokens * q8row_stride(max_d_model));
    rc |= dev_alloc(&c->q8x2, (size_t)max_tokens * q8row_stride(max_d_model));
    rc |= dev_alloc(&c->act, P * max_d_ff);
    rc |= dev_alloc(&c->q8act, P * q8row_stride(max_d_ff));
    rc |= dev_alloc(reinterpret_cast<uint16_t **>(&c->xq_f16), P * max_d_model);
    rc |= dev_alloc(reinterpret_cast<uint16_t **>(&c->actq_f16), P * max_d_ff);
    rc |= dev_alloc(&c->xscale, P);
    rc |= dev_alloc(&c->zero_ids, (size_t)max_tokens);
    rc |= dev_alloc(&c->one_w, (size_t)max_tokens);
    rc |= dev_alloc(&c->gate_s, (size_t)max_tokens);
    rc |= dev_alloc(&c->actscale, P);
    rc |= dev_alloc(&c->ydown, P * max_d_model);
    rc |= dev_alloc(&c->logits, (size_t)max_tokens * max_experts);
    if (max_tokens > ROUTER_TILED_TOKENS) rc |= dev_alloc(&c->logits_part, (size_t)router_part_rows(max_tokens) * max_experts);
    rc |= dev_alloc(&c->ids, P);
    rc |= dev_alloc(&c->weights, P);
    rc |= c->plan.alloc(max_experts, (int)P);
    rc |= dev_alloc(&c->err, 1);
    rc |= dev_alloc(&c->bad, 2);
    rc |= dev_alloc(&c->queue, 4);
    rc |= dev_alloc(&c->ticket, 1 + ROUTER_MAX_GROUPS);
    rc |= dev_alloc(&c->small_bar, 2);
    rc |= dev_alloc(&c->x_stage, (size_t)max_tokens * max_d_model);
    rc |= dev_alloc(&c->out_stage, (size_t)max_tokens * max_d_model);
    rc |= ok(cudaStreamCreateWithFlags(&c->host_stream, cudaStreamNonBlocking));
    rc |= ok(cudaHostAlloc(reinterpret_cast<void **>(&c->err_host), sizeof(int), cudaHostAllocDefault));
    if (!rc) {
        rc |= ok(cudaMemset(c->err, 0, sizeof(int)));
        rc |= ok(cudaMemset(c->bad, 0, 2 * sizeof(int)));
        rc |= ok(cudaMemset(c->queue, 0, 4 * sizeof(int)));
        rc |= ok(cudaMemset(c->ticket, 0, (1 + ROUTER_MAX_GROUPS) * sizeof(unsigned)));
        rc |= ok(cudaMemset(c->small_bar, 0, 2 * sizeof(unsigned)));
        rc |= ok(cudaMemset(c->plan.b.hdr, 0, 4 * sizeof(int)));
        rc |= ok(cudaMemset(c->zero_ids, 0, (size_t)max_tokens * sizeof(int32_t)));
        // 1.0f = 0x3f800000: fill through a host staging vector (done once)
        {
            float *ones = new (std::nothrow) float[max_tokens];
            if (!ones) rc |= ZMOE_ERR_ARG;
            else {
                for (int i = 0; i < max_tokens; ++i) ones[i] = 1.0f;
                rc |= ok(cudaMemcpy(c->one_w, ones, (size_t)max_tokens * sizeof(float), cudaMemcpyHostToDevice));
                delete[] ones;
            }
        }
    }
    if (rc) {
        zmoe_ctx_destroy(c);
        return ZMOE_ERR_CUDA;
    }
    *out = c;
    return ZMOE_OK;
}

void zmoe_ctx_destroy(zmoe_ctx *c) {
    if (!c) return;
    cudaFree(c->zero_ids); cudaFree(c->one_w); cudaFree(c->gate_s);
    cudaFree(c->xq_f16); cudaFree(c->actq_f16); cudaFree(c->xscale); cudaFree(c->actscale);
    cudaFree(c->q8x); cudaFree(c->q8x2); cudaFree(c->act); cudaFree(c->act2); cudaFree(c->q8act); cudaFree(c->ydown);
    cudaFree(c->logits); cudaFree(c->logits_part); cudaFree(c->ids); cudaFree(c->weights); cudaFree(c->err); cudaFree(c->bad); cudaFree(c->queue); cudaFree(c->ticket); cudaFree(c->small_bar);
    cudaFree(c->x_stage); cudaFree(c->out_stage);
    c->plan.release();
    if (c->host_stream) cudaStreamDestroy(c->host_stream);
    if (c->err_host) cudaFreeHost(c->err_host);
    delete c;
}

// geometries, item spaces and tile maps of one set of decode kernels for a layer
static int build_proj(const zmoe_layer_desc &d, bool dual, bool allow_v2, zmoe_layer::Proj *P) {
    int rc = mmid_geometry(d.gate.type, d.d_model, d.d_ff, dual, &P->g_gu, allow_v2);
    if (!rc && !dual) {
        rc = mmid_geometry(d.up.type, d.d_model, d.d_ff, false, &P->g_gate1, allow_v2);
        // the two single projections share one item space: both on the K-chunked kernel (32-row items) or neither
        if (!rc && P->g_gu.v2 != P->g_gate1.v2) {
            rc = mmid_geometry(d.gate.type, d.d_model, d.d_ff, false, &P->g_gu, false);
            if (!rc) rc = mmid_geometry(d.up.type, d.d_model, d.d_ff, false, &P->g_gate1, false);
        }
        if (!rc) {
            // ... with the smaller tile and the fewer pairs per item of the two
            if (P->g_gate1.R < P->g_gu.R) P->g_gu.R = P->g_gate1.R; else P->g_gate1.R = P->g_gu.R;
            const int mt = P->g_gu.maxtok < P->g_gate1.maxtok ? P->g_gu.maxtok : P->g_gate1.maxtok;
            P->g_gu.maxtok = mt; P->g_gate1.maxtok = mt;
        }
    }
    if (!rc) rc = mmid_geometry(d.down.type, d.d_ff, d.d_model, false, &P->g_dn, allow_v2);
    if (rc) return rc;
    P->nrt_gu = (d.d_ff + P->g_gu.R - 1) / P->g_gu.R;
    P->nrt_dn = (d.d_model + P->g_dn.R - 1) / P->g_dn.R;
    P->mt_gu = P->g_gu.maxtok;
    P->mt_dn = P->g_dn.maxtok;
    const int rb_gu = (d.d_model / QK_K) * block_bytes(d.gate.type), rb_dn = (d.d_ff / QK_K) * block_bytes(d.down.type);
    if (P->g_gu.v2) {
        if (P->g_gu.tiled) {
            P->has_tm_gu =
                make_chunk_map(&P->tm_gate, d.gate.data_dev, d.n_experts, d.d_ff, rb_gu, d.gate.expert_stride, P->g_gu.pitch) == ZMOE_OK;
            if (dual)
                P->has_tm_gu = P->has_tm_gu && make_chunk_map(&P->tm_up, d.up.data_dev, d.n_experts, d.d_ff, rb_gu,
                                                              d.up.expert_stride, P->g_gu.pitch) == ZMOE_OK;
            if (!P->has_tm_gu) return ZMOE_ERR_CUDA;
        }
        if (!dual && P->g_gate1.tiled &&
            make_chunk_map(&P->tm_up, d.up.data_dev, d.n_experts, d.d_ff, (d.d_model / QK_K) * block_bytes(d.up.type),
                           d.up.expert_stride, P->g_gate1.pitch) != ZMOE_OK)
            return ZMOE_ERR_CUDA;
    } else if (dual && P->g_gu.rbs != rb_gu) {
        P->has_tm_gu =
            make_rows_map(&P->tm_gate, d.gate.data_dev, d.n_experts, d.d_ff, rb_gu, d.gate.expert_stride, P->g_gu.R) == ZMOE_OK &&
            make_rows_map(&P->tm_up, d.up.data_dev, d.n_experts, d.d_ff, rb_gu, d.up.expert_stride, P->g_gu.R) == ZMOE_OK;
    }
    if (P->g_dn.v2) {
        if (P->g_dn.tiled) {
            P->has_tm_dn = make_chunk_map(&P->tm_down, d.down.data_dev, d.n_experts, d.d_model, rb_dn, d.down.expert_stride,
                                          P->g_dn.pitch) == ZMOE_OK;
            if (!P->has_tm_dn) return ZMOE_ERR_CUDA;
        }
    } else if (P->g_dn.rbs != rb_dn) {
        P->has_tm_dn = make_rows_map(&P->tm_down, d.down.data_dev, d.n_experts, d.d_model, rb_dn, d.down.expert_stride,
                                     P->g_dn.R) == ZMOE_OK;
    }
    return ZMOE_OK;
}

// the same for the integer tensor-core kernel: which of the two item spaces have it
static void build_tc(const zmoe_layer_desc &d, bool dual, zmoe_layer::Proj *P) {
    const int D = d.d_model, F = d.d_ff, E = d.n_experts;
    auto rb = [](int type, int I) { return (I / QK_K) * block_bytes(type); };
    P->has_tm_gu = tc_geometry(d.gate.type, D, F, dual, &P->g_gu) == ZMOE_OK && tc_geometry(d.up.type, D, F, dual, &P->g_gate1) == ZMOE_OK &&
                   make_tc_map(&P->tm_gate, d.gate.data_dev, E, F, rb(d.gate.type, D), d.gate.expert_stride, P->g_gu.pitch, P->g_gu.g_log2) == ZMOE_OK &&
                   make_tc_map(&P->tm_up, d.up.data_dev, E, F, rb(d.up.type, D), d.up.expert_stride, P->g_gate1.pitch, P->g_gate1.g_log2) == ZMOE_OK;
    P->has_tm_dn = tc_geometry(d.down.type, F, D, false, &P->g_dn) == ZMOE_OK &&
                   make_tc_map(&P->tm_down, d.down.data_dev, E, D, rb(d.down.type, F), d.down.expert_stride, P->g_dn.pitch, P->g_dn.g_log2) == ZMOE_OK;
    if (P->has_tm_gu) P->nrt_gu = (F + P->g_gu.R - 1) / P->g_gu.R;
    if (P->has_tm_dn) P->nrt_dn = (D + P->g_dn.R - 1) / P->g_dn.R;
}

int zmoe_layer_create(zmoe_ctx *ctx, const zmoe_layer_desc *desc, zmoe_layer **out) {
    if (!ctx || !desc || !out) return ZMOE_ERR_ARG;
    const zmoe_layer_desc &d = *desc;
    if (d.d_model <= 0 || d.d_ff <= 0 || d.n_experts <= 0 || d.topk <= 0 || d.topk > d.n_experts) return ZMOE_ERR_ARG;
    if (!d.gate.data_dev || !d.up.data_dev || !d.down.data_dev) return ZMOE_ERR_ARG;
    if (d.d_model > ctx->max_d || d.d_ff > ctx->max_f || d.n_experts > ctx->max_e || d.topk > ctx->max_k)
        return ZMOE_ERR_CAPACITY;
    if (d.d_model % QK_K || d.d_ff % QK_K) return ZMOE_ERR_SHAPE;
    zmoe_layer *L = new (std::nothrow) zmoe_layer();
    if (!L) return ZMOE_ERR_ARG;
    L->ctx = ctx;
    L->d = d;
    L->dual = d.gate.type == d.up.type;
    int rc = build_proj(d, L->dual, true, &L->big);
    if (!rc) rc = build_proj(d, L->dual, false, &L->small);
    const zmoe_weight *ws[3] = {&d.gate, &d.up, &d.down};
    size_t *tot[3] = {&L->bytes_gate, &L->bytes_up, &L->bytes_down};
    for (int i = 0; i < 3 && !rc; ++i) {
        const int I = i < 2 ? d.d_model : d.d_ff, O = i < 2 ? d.d_ff : d.d_model;
        const size_t need = (size_t)O * (I / QK_K) * block_bytes(ws[i]->type);
        if (ws[i]->expert_stride < need) rc = ZMOE_ERR_ARG;
        if ((reinterpret_cast<size_t>(ws[i]->data_dev) & 15) || (ws[i]->expert_stride & 15)) rc = ZMOE_ERR_ALIGN;
        const size_t end = (size_t)(d.n_experts - 1) * ws[i]->expert_stride + need;
        *tot[i] = ws[i]->bytes ? ws[i]->bytes : end;
        if (*tot[i] < end) L->whole = false;
    }
    if (!rc && !L->dual && !ctx->act2)
        rc = dev_alloc(&ctx->act2, (size_t)2 * ctx->max_t * ctx->max_k * ctx->max_f);
    if (rc) {
        delete L;
        return rc;
    }
    build_tc(d, L->dual, &L->tc);
    L->gemm_shape = L->dual && gemm_sm100_supported(d.gate.type, d.d_model, d.d_ff) && gemm_sm100_supported(d.down.type, d.d_ff, d.d_model) &&
                    d.n_experts <= 512;
    *out = L;
    return ZMOE_OK;
}

void zmoe_layer_destroy(zmoe_layer *layer) { delete layer; }

// whether zmoe_expert_ffn will take the tensor-core grouped GEMM for T tokens (the rule of the header:
// shapes allow it, and the path is forced to 2 or left at 0 with enough pairs per expert)
static bool takes_gemm(const zmoe_layer *L, int T) {
    const int path = L->ctx->path;
    return L->gemm_shape && (path == 2 || (path == 0 && (long)T * L->d.topk >= (long)kGemmMinPairsPerExpert * L->d.n_experts)) &&
           gemm_sm100_built(L->d.gate.type) && gemm_sm100_built(L->d.down.type);
}

// how the quantiser writes rows that meet weights of `type`
static int q8_rows_for(int type, bool on_tc) { return q8_layout_of(type) | (on_tc ? Q8_FOR_TC : 0); }

// packed Q8_K rows of the layer input for the decode kernels (both unit layouts where gate and up differ)
static int quantize_input(zmoe_layer *L, const float *x_dev, int T, bool on_tc, cudaStream_t st) {
    zmoe_ctx *c = L->ctx;
    int rc = launch_quantize_rows(x_dev, L->d.d_model, c->q8x, T, L->d.d_model, q8_rows_for(L->d.gate.type, on_tc), st);
    g_launches += 1;
    if (!rc && q8_layout_of(L->d.up.type) != q8_layout_of(L->d.gate.type)) {
        rc = launch_quantize_rows(x_dev, L->d.d_model, c->q8x2, T, L->d.d_model, q8_rows_for(L->d.up.type, on_tc), st);
        g_launches += 1;
    }
    if (!rc) c->q8x_valid = true;
    return rc;
}

// the arguments of a router launch for T tokens whose plan is built for the kernels cg
static RouterArgs router_args(const zmoe_layer *L, const float *x_dev, int T, const CallGeom &cg) {
    const zmoe_ctx *c = L->ctx;
    RouterArgs a;
    a.x = x_dev; a.wr = L->d.router_w_dev; a.bias = L->d.router_bias_dev;
    a.T = T; a.D = L->d.d_model; a.E = L->d.n_experts; a.K = L->d.topk;
    a.gating = L->d.gating; a.normalize = L->d.weights_norm;
    a.weight_scale = L->d.weights_scale;
    a.n_groups = L->d.n_groups; a.n_groups_used = L->d.n_groups_used;
    a.logits = c->logits; a.ids = c->ids; a.weights = c->weights; a.q8x = c->q8x;
    a.plan = c->plan.b;
    a.stats = gemm_stats_buffer(0);
    a.q8_layout = q8_rows_for(L->d.gate.type, cg.gu == SET_TC);
    a.plan.mt_gu = cg.mt_gu; a.plan.mt_dn = cg.mt_dn;
    a.nrt_gu = cg.nrt_gu; a.nrt_dn = cg.nrt_dn;
    a.ticket = c->ticket;
    a.logits_part = c->logits_part;
    a.logits_part_rows = router_part_rows(c->max_t) * c->max_e / L->d.n_experts;
    a.n_sm = c->n_sm;
    return a;
}

int zmoe_route(zmoe_layer *L, const float *x_dev, int T, void *stream) {
    if (!L || !x_dev || T <= 0) return ZMOE_ERR_ARG;
    zmoe_ctx *c = L->ctx;
    if (T > c->max_t) return ZMOE_ERR_CAPACITY;
    if (!L->d.router_w_dev) return ZMOE_ERR_STATE;
    const CallGeom cg = call_geom(L, T, c->path);
    RouterArgs a = router_args(L, x_dev, T, cg);
    const bool big = router_takes_tiles(T, a.D, a.E);
    // the tensor-core path quantises the rows itself while it gathers them: the large-batch router then skips q8x
    a.want_q8x = !(big && takes_gemm(L, T));
    int rc = big ? launch_router_prefill(a, static_cast<cudaStream_t>(stream))
                 : launch_router_decode(a, static_cast<cudaStream_t>(stream));
    g_launches += big ? (a.want_q8x ? 4 : 3) : 1;
    c->q8x_valid = a.want_q8x;
    if (!rc && a.want_q8x && q8_layout_of(L->d.up.type) != q8_layout_of(L->d.gate.type)) {
        rc = launch_quantize_rows(x_dev, L->d.d_model, c->q8x2, T, L->d.d_model, q8_rows_for(L->d.up.type, cg.gu == SET_TC),
                                  static_cast<cudaStream_t>(stream));
        g_launches += 1;
    }
    c->planned = cg;
    if (!rc) { c->routed_t = T; c->x_last = x_dev; }
    return rc;
}

static int set_routes_impl(zmoe_layer *L, const float *x_dev, const int32_t *ids_dev, const float *weights_dev, int T,
                           int first_expert, bool window, void *stream, int ids_ld = 0, int w_ld = 0) {
    if (!L || !x_dev || !ids_dev || !weights_dev || T <= 0) return ZMOE_ERR_ARG;
    zmoe_ctx *c = L->ctx;
    if (T > c->max_t) return ZMOE_ERR_CAPACITY;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t P = (size_t)T * L->d.topk;
    int rc = 0;
    c->q8x_valid = false;
    const CallGeom cg = call_geom(L, T, c->path);
    if (!takes_gemm(L, T)) rc = quantize_input(L, x_dev, T, cg.gu == SET_TC, st);   // the tensor-core path quantises while it gathers
    // the planner takes the routes in (copy, window mapping) before it groups them: one launch
    PlanBuffers pb = c->plan.b;
    pb.mt_gu = cg.mt_gu; pb.mt_dn = cg.mt_dn;
    if (!rc) c->planned = cg;
    if (!rc)
        rc = launch_plan_ingest(ids_dev, weights_dev, c->ids, c->weights, (int)P, L->d.n_experts, first_expert, window,
                                pb, cg.nrt_gu, cg.nrt_dn, st, ids_ld ? L->d.topk : 0, ids_ld, w_ld);
    if (!rc) { g_launches += 1; c->routed_t = T; c->x_last = x_dev; }
    return rc;
}

int zmoe_set_routes(zmoe_layer *L, const float *x_dev, const int32_t *ids_dev, const float *weights_dev, int T,
                    void *stream) {
    return set_routes_impl(L, x_dev, ids_dev, weights_dev, T, 0, false, stream);
}

int zmoe_set_routes_window(zmoe_layer *L, const float *x_dev, const int32_t *ids_dev, const float *weights_dev, int T,
                           int first_expert, void *stream) {
    if (first_expert < 0) return ZMOE_ERR_ARG;
    return set_routes_impl(L, x_dev, ids_dev, weights_dev, T, first_expert, true, stream);
}

int zmoe_set_routes_strided(zmoe_layer *L, const float *x_dev, const int32_t *ids_dev, size_t ids_token_stride,
                            const float *weights_dev, size_t weights_token_stride, int T, void *stream) {
    if (!L) return ZMOE_ERR_ARG;
    const size_t k4 = (size_t)L->d.topk * 4;
    if (ids_token_stride % 4 || weights_token_stride % 4 || ids_token_stride < k4 || weights_token_stride < k4 ||
        ids_token_stride / 4 > INT32_MAX || weights_token_stride / 4 > INT32_MAX)
        return ZMOE_ERR_ALIGN;
    return set_routes_impl(L, x_dev, ids_dev, weights_dev, T, 0, false, stream, (int)(ids_token_stride / 4),
                           (int)(weights_token_stride / 4));
}

int zmoe_expert_ffn(zmoe_layer *L, float *out_dev, int T, int accumulate, void *stream) {
    return zmoe_expert_ffn_events(L, out_dev, T, accumulate, stream, nullptr, nullptr);
}

int zmoe_expert_ffn_events(zmoe_layer *L, float *out_dev, int T, int accumulate, void *stream, void *ev_before,
                           void *ev_after) {
    if (!L || !out_dev || T <= 0) return ZMOE_ERR_ARG;
    zmoe_ctx *c = L->ctx;
    if (c->routed_t != T) return ZMOE_ERR_STATE;
    if (c->path == 2 && L->gemm_shape && !takes_gemm(L, T)) return ZMOE_ERR_CUDA;   // asked for, and lost in the build: not another kernel without a word
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const zmoe_layer_desc &d = L->d;
    const int P = T * d.topk;
    MmidLaunch m;
    m.plan = c->plan.b;
    m.err = c->err;
    m.bad = c->bad;
    m.queue = c->queue;
    m.n_sm = c->n_sm;
    m.clamp = d.swiglu_clamp;
    m.clamp_fused = d.swiglu_clamp_fused;
    m.multi = T > 1 && c->path != 3;
    int rc;
    // many pairs per expert: the contraction is compute-bound and goes to the tensor cores
    const bool use_gemm = c->x_last && takes_gemm(L, T);
    if (use_gemm) {
        if (ev_before) cudaEventRecord(static_cast<cudaEvent_t>(ev_before), st);
        GemmLaunch g;
        g.plan = c->plan.b; g.err = c->err; g.bad = c->bad; g.n_sm = c->n_sm;
        g.clamp = d.swiglu_clamp; g.clamp_fused = d.swiglu_clamp_fused;
        g.n_experts = d.n_experts;
        rc = launch_q8_roundtrip_tokens_f16(c->x_last, d.d_model, c->xq_f16, c->xscale, c->plan.b, T, d.topk, d.d_model, st);
        g.type = d.gate.type; g.dual = true;
        g.w0 = d.gate.data_dev; g.w1 = d.up.data_dev;
        g.stride0 = d.gate.expert_stride; g.stride1 = d.up.expert_stride;
        g.I = d.d_model; g.O = d.d_ff;
        g.x_f16 = c->xq_f16; g.xscale = c->xscale; g.x_rows = c->max_t * c->max_k;
        g.y = c->act; g.ldy = d.d_ff;
        if (!rc) rc = launch_gemm_sm100(g, st);
        if (ev_after) cudaEventRecord(static_cast<cudaEvent_t>(ev_after), st);
        if (!rc) rc = launch_q8_roundtrip_f16(c->act, d.d_ff, c->actq_f16, c->actscale, c->plan.b, P, 1, d.d_ff, st);
        g.type = d.down.type; g.dual = false;
        g.w0 = d.down.data_dev; g.w1 = nullptr;
        g.stride0 = d.down.expert_stride; g.stride1 = 0;
        g.I = d.d_ff; g.O = d.d_model;
        g.x_f16 = c->actq_f16; g.xscale = c->actscale; g.x_rows = c->max_t * c->max_k;
        g.y = c->ydown; g.ldy = d.d_model;
        if (!rc) rc = launch_gemm_sm100(g, st);
        if (!rc) rc = launch_combine(out_dev, c->ydown, c->weights, c->ids, T, d.topk, d.d_model, d.n_experts, accumulate, st);
        g_launches += 5;
        return rc;
    }
    // the path may have been changed since the routes were set: the decode kernels need the quantised input
    if (!plan_fits(L, T, c->planned)) {
        // the routes were made through another layer of this context, whose items or rows are not this one's
        c->planned = call_geom(L, T, c->path);
        c->q8x_valid = false;
        m.plan.mt_gu = c->planned.mt_gu; m.plan.mt_dn = c->planned.mt_dn;
        rc = launch_plan_from_ids(c->ids, P, d.n_experts, m.plan, c->planned.nrt_gu, c->planned.nrt_dn, st);
        if (rc) return rc;
        g_launches += 1;
    }
    if (!c->q8x_valid) {
        if (!c->x_last) return ZMOE_ERR_STATE;
        rc = quantize_input(L, c->x_last, T, c->planned.gu == SET_TC, st);
        if (rc) return rc;
    }
    m.plan.mt_gu = c->planned.mt_gu; m.plan.mt_dn = c->planned.mt_dn;
    const zmoe_layer::Proj &ps = L->set(c->planned.gu), &pd = L->set(c->planned.dn);
    if (ev_before) cudaEventRecord(static_cast<cudaEvent_t>(ev_before), st);
    if (L->dual) {
        m.type = d.gate.type; m.dual = true;
        m.w0 = d.gate.data_dev; m.w1 = d.up.data_dev;
        m.stride0 = d.gate.expert_stride; m.stride1 = d.up.expert_stride;
        m.total0 = L->bytes_gate; m.total1 = L->bytes_up;
        m.I = d.d_model; m.O = d.d_ff;
        m.q8 = c->q8x; m.xdiv = d.topk;
        m.y = c->act; m.ldy = d.d_ff;
        m.down = false;
        if (ps.has_tm_gu) { m.tm0 = &ps.tm_gate; m.tm1 = &ps.tm_up; }
        rc = launch_mmid(m, ps.g_gu, st);
        m.tm0 = nullptr; m.tm1 = nullptr;
        g_launches += 1;
    } else {
        float *gbuf = c->act2, *ubuf = c->act2 + (size_t)P * d.d_ff;
        m.dual = false; m.w1 = nullptr; m.stride1 = 0; m.total1 = 0;
        m.I = d.d_model; m.O = d.d_ff; m.q8 = c->q8x; m.xdiv = d.topk; m.ldy = d.d_ff; m.down = false;
        m.type = d.up.type; m.w0 = d.up.data_dev; m.stride0 = d.up.expert_stride; m.total0 = L->bytes_up; m.y = ubuf;
        if (q8_layout_of(d.up.type) != q8_layout_of(d.gate.type)) m.q8 = c->q8x2;
        m.tm0 = ps.g_gate1.tc || (ps.g_gate1.v2 && ps.g_gate1.tiled) ? &ps.tm_up : nullptr;
        rc = launch_mmid(m, ps.g_gate1, st);
        m.q8 = c->q8x;
        m.type = d.gate.type; m.w0 = d.gate.data_dev; m.stride0 = d.gate.expert_stride; m.total0 = L->bytes_gate; m.y = gbuf;
        m.tm0 = ps.g_gu.tc || (ps.g_gu.v2 && ps.g_gu.tiled) ? &ps.tm_gate : nullptr;
        if (!rc) rc = launch_mmid(m, ps.g_gu, st);
        m.tm0 = nullptr;
        if (!rc) {
            launch_expert_swiglu(c->act, gbuf, ubuf, P * d.d_ff, d.swiglu_clamp, d.swiglu_clamp_fused, c->bad, stream);
            rc = ok(cudaPeekAtLastError());
        }
        g_launches += 3;
    }
    if (ev_after) cudaEventRecord(static_cast<cudaEvent_t>(ev_after), st);
    if (!rc) rc = launch_quantize_rows(c->act, d.d_ff, c->q8act, P, d.d_ff, q8_rows_for(d.down.type, c->planned.dn == SET_TC), st);
    if (!rc) {
        m.type = d.down.type; m.dual = false;
        m.w0 = d.down.data_dev; m.w1 = nullptr;
        m.stride0 = d.down.expert_stride; m.stride1 = 0;
        m.total0 = L->bytes_down; m.total1 = 0;
        m.I = d.d_ff; m.O = d.d_model;
        m.q8 = c->q8act; m.xdiv = 1;
        m.y = c->ydown; m.ldy = d.d_model;
        m.down = true;
        if (pd.has_tm_dn) m.tm0 = &pd.tm_down;
        rc = launch_mmid(m, pd.g_dn, st);
    }
    if (!rc) rc = launch_combine(out_dev, c->ydown, c->weights, c->ids, T, d.topk, d.d_model, d.n_experts, accumulate, st);
    g_launches += 3;
    return rc;
}

int zmoe_dense_ffn(zmoe_layer *L, const float *x_dev, float *out_dev, int T, int accumulate, void *stream) {
    if (!L || !x_dev || !out_dev || T <= 0) return ZMOE_ERR_ARG;
    if (L->d.n_experts != 1 || L->d.topk != 1) return ZMOE_ERR_STATE;
    if (T > L->ctx->max_t) return ZMOE_ERR_CAPACITY;
    int rc = zmoe_set_routes(L, x_dev, L->ctx->zero_ids, L->ctx->one_w, T, stream);
    if (!rc) rc = zmoe_expert_ffn(L, out_dev, T, accumulate, stream);
    return rc;
}

int zmoe_dense_ffn_gated(zmoe_layer *L, const float *x_dev, const float *gate_w_dev, float *out_dev, int T, int accumulate,
                         void *stream) {
    if (!L || !x_dev || !gate_w_dev || !out_dev || T <= 0) return ZMOE_ERR_ARG;
    if (L->d.n_experts != 1 || L->d.topk != 1) return ZMOE_ERR_STATE;
    if (T > L->ctx->max_t) return ZMOE_ERR_CAPACITY;
    // the scalar gate rides as the route weight: the combine multiplies each token's row by it
    int rc = launch_token_gate(x_dev, gate_w_dev, L->ctx->gate_s, T, L->d.d_model, static_cast<cudaStream_t>(stream));
    g_launches += 1;
    if (!rc) rc = zmoe_set_routes(L, x_dev, L->ctx->zero_ids, L->ctx->gate_s, T, stream);
    if (!rc) rc = zmoe_expert_ffn(L, out_dev, T, accumulate, stream);
    return rc;
}

int zmoe_moe_forward(zmoe_layer *L, const float *x_dev, float *out_dev, int T, void *stream) {
    return zmoe::layer_forward(L, x_dev, out_dev, T, 0, stream);
}

int zmoe_moe_forward_bf16(zmoe_layer *L, const void *x_bf16_dev, float *out_dev, int T, void *stream) {
    if (!L || !x_bf16_dev || !out_dev || T <= 0) return ZMOE_ERR_ARG;
    zmoe_ctx *c = L->ctx;
    if (T > c->max_t) return ZMOE_ERR_CAPACITY;
    // widened once into the context's staging rows (exact); router and matmuls then read f32 as ever
    int rc = launch_widen_bf16(x_bf16_dev, c->x_stage, (long)T * L->d.d_model, c->n_sm, static_cast<cudaStream_t>(stream));
    g_launches += 1;
    if (!rc) rc = zmoe_moe_forward(L, c->x_stage, out_dev, T, stream);
    return rc;
}

int zmoe_moe_forward_host(zmoe_layer *L, const float *x_host, float *out_host, int T) {
    if (!L || !x_host || !out_host || T <= 0) return ZMOE_ERR_ARG;
    zmoe_ctx *c = L->ctx;
    if (T > c->max_t) return ZMOE_ERR_CAPACITY;
    const size_t n = (size_t)T * L->d.d_model * sizeof(float);
    int rc = ok(cudaMemcpyAsync(c->x_stage, x_host, n, cudaMemcpyHostToDevice, c->host_stream));
    if (!rc) rc = zmoe_moe_forward(L, c->x_stage, c->out_stage, T, c->host_stream);
    if (!rc) rc = ok(cudaMemcpyAsync(out_host, c->out_stage, n, cudaMemcpyDeviceToHost, c->host_stream));
    // the device error flag rides on the same stream: one synchronisation for output and status
    if (!rc) rc = ok(cudaMemcpyAsync(c->err_host, c->err, sizeof(int), cudaMemcpyDeviceToHost, c->host_stream));
    if (!rc) rc = ok(cudaStreamSynchronize(c->host_stream));
    if (!rc && *c->err_host) {
        cudaMemset(c->err, 0, sizeof(int));
        cudaMemset(c->queue, 0, 4 * sizeof(int));   // a launch that gave up may have left its tickets behind
        cudaMemset(c->small_bar, 0, 2 * sizeof(unsigned));
        rc = ZMOE_ERR_DEVICE_WAIT;
    }
    return rc;
}

int zmoe_get_routes(zmoe_ctx *c, int T, int topk, int32_t *ids_host, float *weights_host) {
    if (!c || T <= 0 || topk <= 0 || (size_t)T * topk > (size_t)c->max_t * c->max_k) return ZMOE_ERR_ARG;
    int rc = 0;
    if (ids_host) rc |= ok(cudaMemcpy(ids_host, c->ids, (size_t)T * topk * sizeof(int32_t), cudaMemcpyDeviceToHost));
    if (weights_host) rc |= ok(cudaMemcpy(weights_host, c->weights, (size_t)T * topk * sizeof(float), cudaMemcpyDeviceToHost));
    return rc ? ZMOE_ERR_CUDA : ZMOE_OK;
}

int zmoe_copy_routes(zmoe_ctx *c, int T, int topk, int32_t *ids_dev, float *weights_dev, void *stream) {
    if (!c || T <= 0 || topk <= 0 || (size_t)T * topk > (size_t)c->max_t * c->max_k) return ZMOE_ERR_ARG;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int rc = 0;
    if (ids_dev) rc |= ok(cudaMemcpyAsync(ids_dev, c->ids, (size_t)T * topk * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
    if (weights_dev) rc |= ok(cudaMemcpyAsync(weights_dev, c->weights, (size_t)T * topk * sizeof(float), cudaMemcpyDeviceToDevice, st));
    return rc ? ZMOE_ERR_CUDA : ZMOE_OK;
}

int zmoe_get_expert_freq(zmoe_ctx *c, int n_experts, int32_t *freq_host) {
    if (!c || !freq_host || n_experts <= 0 || n_experts > c->max_e) return ZMOE_ERR_ARG;
    return ok(cudaMemcpy(freq_host, c->plan.b.freq, (size_t)n_experts * sizeof(int32_t), cudaMemcpyDeviceToHost));
}

int zmoe_get_probs(zmoe_ctx *c, int T, int n_experts, float *probs_host) {
    if (!c || !probs_host || T <= 0 || (size_t)T * n_experts > (size_t)c->max_t * c->max_e) return ZMOE_ERR_ARG;
    return ok(cudaMemcpy(probs_host, c->logits, (size_t)T * n_experts * sizeof(float), cudaMemcpyDeviceToHost));
}

int zmoe_get_act(zmoe_ctx *c, int n_pairs, int d_ff, float *act_host) {
    if (!c || !act_host || n_pairs <= 0 || (size_t)n_pairs * d_ff > (size_t)c->max_t * c->max_k * c->max_f) return ZMOE_ERR_ARG;
    return ok(cudaMemcpy(act_host, c->act, (size_t)n_pairs * d_ff * sizeof(float), cudaMemcpyDeviceToHost));
}

int zmoe_ctx_set_path(zmoe_ctx *c, int path) {
    if (!c || path < 0 || path > 3) return ZMOE_ERR_ARG;
    c->path = path;
    return ZMOE_OK;
}

int zmoe_ctx_check(zmoe_ctx *c) {
    if (!c) return ZMOE_ERR_ARG;
    int e = 0;
    if (cudaMemcpy(&e, c->err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return ZMOE_ERR_CUDA;
    if (e) {
        cudaMemset(c->err, 0, sizeof(int));
        cudaMemset(c->queue, 0, 4 * sizeof(int));   // a launch that gave up may have left its tickets behind
        cudaMemset(c->small_bar, 0, 2 * sizeof(unsigned));
        return ZMOE_ERR_DEVICE_WAIT;
    }
    return ZMOE_OK;
}

int zmoe_ctx_bad_counts(zmoe_ctx *c, int32_t *counts_host, int clear) {
    if (!c || !counts_host) return ZMOE_ERR_ARG;
    if (cudaMemcpy(counts_host, c->bad, 2 * sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return ZMOE_ERR_CUDA;
    if (clear && (counts_host[0] | counts_host[1]) && cudaMemset(c->bad, 0, 2 * sizeof(int)) != cudaSuccess)
        return ZMOE_ERR_CUDA;
    return ZMOE_OK;
}

int zmoe_gemm_min_pairs_per_expert(void) { return kGemmMinPairsPerExpert; }

int zmoe_debug_gemm_cycles(uint64_t *counters32_host) {
    if (!counters32_host) return ZMOE_ERR_ARG;
    if (cudaDeviceSynchronize() != cudaSuccess) return ZMOE_ERR_CUDA;
    return gemm_stats_read(reinterpret_cast<unsigned long long *>(counters32_host));
}

uint64_t zmoe_kernel_launches(void) { return g_launches.load(); }

}  // extern "C"

bool zmoe::layer_small_args(zmoe_layer *L, const float *x_dev, float *out_dev, int T, int accumulate, RouterArgs *r, SmallLaunch *s) {
    const zmoe_layer_desc &d = L->d;
    if (T > L->ctx->max_t || !d.router_w_dev || !L->dual || !L->whole || !takes_fused(d, T) ||
        !moe_small_supported(d.gate.type, d.down.type, T, d.d_model, d.d_ff, d.n_experts, d.topk))
        return false;
    zmoe_ctx *c = L->ctx;
    *r = router_args(L, x_dev, T, call_geom(L, T, 0));
    s->type_gu = d.gate.type; s->type_dn = d.down.type; s->F = d.d_ff;
    s->w_gate = d.gate.data_dev; s->w_up = d.up.data_dev; s->w_down = d.down.data_dev;
    s->stride_gate = d.gate.expert_stride; s->stride_up = d.up.expert_stride; s->stride_down = d.down.expert_stride;
    s->clamp = d.swiglu_clamp; s->clamp_fused = d.swiglu_clamp_fused;
    s->act = c->act; s->out = out_dev; s->accumulate = accumulate;
    s->err = c->err; s->bad = c->bad; s->bar = c->small_bar;
    return true;
}

void zmoe::layer_small_done(zmoe_layer *L, const float *x_dev, int T) {
    zmoe_ctx *c = L->ctx;
    c->planned = call_geom(L, T, 0);
    c->q8x_valid = true;
    c->routed_t = T;
    c->x_last = x_dev;
}

int zmoe::layer_forward(zmoe_layer *L, const float *x_dev, float *out_dev, int T, int accumulate, void *stream) {
    RouterArgs r;
    SmallLaunch s;
    if (L && x_dev && out_dev && T > 0 && L->ctx->path < 2 && repeats_little(L->d, T) && layer_small_args(L, x_dev, out_dev, T, accumulate, &r, &s)) {
        const int rc = launch_moe_small(r, s, static_cast<cudaStream_t>(stream));
        if (!rc) {
            g_launches += 1;
            layer_small_done(L, x_dev, T);
        }
        if (rc != ZMOE_ERR_STATE) return rc;
    }
    int rc = zmoe_route(L, x_dev, T, stream);
    if (!rc) rc = zmoe_expert_ffn(L, out_dev, T, accumulate, stream);
    return rc;
}

// ---------------------------------------------------------------------------
// per-device scratch of the handle-free entry points
// ---------------------------------------------------------------------------
namespace {

struct DeviceScratch {
    uint8_t *q8 = nullptr;
    size_t q8_bytes = 0;
    PlanStore plan;
    int *err = nullptr;
    int32_t *ids = nullptr;
    size_t ids_cap = 0;
    int n_sm = 0;
};
constexpr int kMaxDevices = 64;
DeviceScratch g_scratch[kMaxDevices];
std::mutex g_scratch_mu;

using ScratchLock = std::unique_lock<std::mutex>;

// Makes sure the current device's scratch can hold `rows` packed rows of I elements, a plan for E experts
// and P pairs, and hands it out LOCKED: the caller keeps `lock` until its kernels are enqueued, so no other
// host thread can grow (free and reallocate) the buffers between this call's launches.  Growing waits for
// the device first, so kernels already enqueued never see a freed buffer.
int scratch_get(int rows, int I, int E, int P, DeviceScratch **out, ScratchLock &lock) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return ZMOE_ERR_CUDA;
    lock = ScratchLock(g_scratch_mu);
    DeviceScratch &s = g_scratch[dev];
    if (!s.n_sm) s.n_sm = sm_count();
    const size_t need = (size_t)rows * q8row_stride(I);
    if (need > s.q8_bytes) {
        if (s.q8) { cudaDeviceSynchronize(); cudaFree(s.q8); }
        if (dev_alloc(&s.q8, need)) return ZMOE_ERR_CUDA;
        s.q8_bytes = need;
    }
    if (E > s.plan.cap_e || P > s.plan.cap_p) {
        const int ne = E > s.plan.cap_e ? E : s.plan.cap_e, np = P > s.plan.cap_p ? P : s.plan.cap_p;
        if (s.plan.cap_e) { cudaDeviceSynchronize(); s.plan.release(); }
        if (s.plan.alloc(ne, np)) return ZMOE_ERR_CUDA;
    }
    if ((size_t)P > s.ids_cap) {
        if (s.ids) { cudaDeviceSynchronize(); cudaFree(s.ids); }
        if (dev_alloc(&s.ids, (size_t)P)) return ZMOE_ERR_CUDA;
        s.ids_cap = P;
    }
    if (!s.err) {
        if (dev_alloc(&s.err, 1)) return ZMOE_ERR_CUDA;
        cudaMemset(s.err, 0, sizeof(int));
    }
    *out = &s;
    return ZMOE_OK;
}

int dense_matmul(int type, float *y, const float *x, int ldx, const void *w, int S, int I, int O, int ldy,
                 cudaStream_t st) {
    if (!y || !x || !w || S <= 0 || I <= 0 || O <= 0) return ZMOE_ERR_ARG;
    MmidGeom g;
    int rc = mmid_geometry(type, I, O, false, &g);
    if (rc) return rc;
    DeviceScratch *s;
    ScratchLock lock;
    rc = scratch_get(S, I, 1, S, &s, lock);
    if (rc) return rc;
    const int nrt = (O + g.R - 1) / g.R;
    rc = launch_quantize_rows(x, ldx, s->q8, S, I, q8_layout_of(type), st);
    if (!rc) rc = launch_plan_dense(S, s->plan.b, nrt, st);
    if (rc) return rc;
    MmidLaunch m;
    m.type = type; m.dual = false;
    m.w0 = w; m.w1 = nullptr;
    m.stride0 = 0; m.stride1 = 0;
    m.total0 = (size_t)O * (I / QK_K) * block_bytes(type); m.total1 = 0;
    m.I = I; m.O = O;
    m.q8 = s->q8; m.xdiv = 1;
    m.y = y; m.ldy = ldy;
    m.plan = s->plan.b;
    m.down = false;
    m.clamp = 0.f; m.clamp_fused = 0;
    m.err = s->err;
    m.n_sm = s->n_sm;
    m.multi = S > 1;
    rc = launch_mmid(m, g, st);
    g_launches += 3;
    return rc;
}

// rows of y whose expert id is >= E become NaN (ids < 0 stay zero)
__global__ void fill_bad_rows_kernel(float *y, int ldy, const int32_t *ids, int P, int E, int O) {
    const int p = blockIdx.x;
    if (p >= P || ids[p] < E) return;
    for (int o = threadIdx.x; o < O; o += blockDim.x) y[(size_t)p * ldy + o] = nanf("");
}
void fill_bad_rows(float *y, int ldy, const int32_t *ids, int P, int E, int O, cudaStream_t st) {
    fill_bad_rows_kernel<<<P, 128, 0, st>>>(y, ldy, ids, P, E, O);
}

// One warp waits, with a short limit, on a barrier that nobody arrives on: the wait runs out, the warp raises
// the error word exactly as the matmul kernels do, and returns.  Exists so that the path from an expired
// device-side wait to ZMOE_ERR_DEVICE_WAIT can be exercised without a hang or a fault.
__global__ void wait_expiry_probe_kernel(int *err) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_init_fence();
    }
    __syncwarp();
    if (!mbar_wait(&bar, 0, 256) && threadIdx.x == 0) atomicExch(err, 1);
}

__global__ void gather_ids_kernel(const uint8_t *src, size_t nb0, size_t nb1, int32_t *dst, int K, int T) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= K * T) return;
    const int t = i / K, k = i % K;
    dst[i] = *reinterpret_cast<const int32_t *>(src + t * nb1 + k * nb0);
}

}  // namespace

extern "C" {

int zmoe_reserve(int rows, int I) {
    if (rows <= 0 || I <= 0 || I % QK_K) return ZMOE_ERR_ARG;
    DeviceScratch *s;
    ScratchLock lock;
    return scratch_get(rows, I, 1, rows, &s, lock);
}

int zmoe_last_status(void) { return tl_status; }

int zmoe_device_status(void) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return ZMOE_ERR_CUDA;
    if (cudaDeviceSynchronize() != cudaSuccess) return ZMOE_ERR_CUDA;
    int seen = 0;
    {
        ScratchLock lock(g_scratch_mu);
        DeviceScratch &s = g_scratch[dev];
        if (s.err) {
            int e = 0;
            if (cudaMemcpy(&e, s.err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return ZMOE_ERR_CUDA;
            if (e) {
                seen = e;
                if (cudaMemset(s.err, 0, sizeof(int)) != cudaSuccess) return ZMOE_ERR_CUDA;
            }
        }
    }
    int e2 = 0;
    if (noalloc_take_error(&e2)) return ZMOE_ERR_CUDA;
    return (seen || e2) ? ZMOE_ERR_DEVICE_WAIT : ZMOE_OK;
}

int zmoe_selftest_wait_expiry(void *stream) {
    DeviceScratch *s;
    ScratchLock lock;
    int rc = scratch_get(1, QK_K, 1, 1, &s, lock);
    if (rc) return rc;
    wait_expiry_probe_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(s->err);
    g_launches += 1;
    return ok(cudaPeekAtLastError());
}

#define ZMOE_DENSE(name, type)                                                                         \
    void name##_stream(float *y, const float *x, const void *w, int S, int I, int O, void *stream) {     \
        tl_status = dense_matmul(type, y, x, I, w, S, I, O, O, static_cast<cudaStream_t>(stream));      \
    }                                                                                                    \
    void name(float *y, const float *x, const void *w, int S, int I, int O) {                            \
        tl_status = dense_matmul(type, y, x, I, w, S, I, O, O, nullptr);                                \
    }

ZMOE_DENSE(launch_q2_K_matmul, Q2_K)
ZMOE_DENSE(launch_q3_K_matmul, Q3_K)
ZMOE_DENSE(launch_q4_K_matmul, Q4_K)
ZMOE_DENSE(launch_iq2_xxs_matmul, IQ2_XXS)

bool zmoe_f32_quant_hook(const zmoe_tensor *w, const zmoe_tensor *x, const zmoe_tensor *ids,
                         zmoe_tensor *y, void *stream, bool execute) {
    constexpr int GGML_F32 = 0, GGML_I32 = 26;
    if (!w || !x || !y || block_bytes(w->type) == 0 || x->type != GGML_F32 || y->type != GGML_F32 || w->ne[0] <= 0 ||
        w->ne[0] > INT32_MAX || w->ne[1] <= 0 || w->ne[1] > INT32_MAX || w->ne[0] % 256 || x->nb[0] != sizeof(float) ||
        y->nb[0] != sizeof(float))
        return false;
    const int I = (int)w->ne[0], O = (int)w->ne[1];
    const size_t row = (size_t)(I / 256) * block_bytes(w->type);
    if (w->nb[1] != row || x->ne[0] != I || y->ne[0] != O) return false;
    MmidGeom g;
    if (mmid_geometry(w->type, I, O, false, &g) != ZMOE_OK) return false;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (ids) {
        if (ids->type != GGML_I32 || ids->nb[0] != sizeof(int32_t) || ids->ne[0] <= 0 || ids->ne[0] > 65535 ||
            ids->ne[1] <= 0 || ids->ne[1] > 65535 || w->ne[2] <= 0 || w->ne[2] > INT32_MAX || w->ne[3] != 1 ||
            (x->ne[1] != 1 && x->ne[1] != ids->ne[0]) || x->ne[2] != ids->ne[1] || x->ne[3] != 1 ||
            y->ne[1] != ids->ne[0] || y->ne[2] != ids->ne[1] || y->ne[3] != 1)
            return false;
        const int K = (int)ids->ne[0], T = (int)ids->ne[1], E = (int)w->ne[2];
        const int xr = (int)x->ne[1];
        // rows of x and y must form one evenly strided list of pairs
        if (x->nb[1] % 4 || x->nb[2] % 4 || y->nb[1] % 4) return false;
        if (xr != 1 && x->nb[2] != (size_t)xr * x->nb[1]) return false;
        if (y->nb[2] != (size_t)K * y->nb[1]) return false;
        if ((reinterpret_cast<size_t>(w->data) & 15) || (w->nb[2] & 15)) return false;
        if (!execute) return true;
        DeviceScratch *s;
        ScratchLock lock;
        const int rows = T * xr;
        if (scratch_get(rows, I, E, K * T, &s, lock)) return false;
        const int ldx = xr == 1 ? (int)(x->nb[2] / 4) : (int)(x->nb[1] / 4);
        int rc = launch_quantize_rows(static_cast<const float *>(x->data), ldx, s->q8, rows, I, q8_layout_of(w->type), st);
        gather_ids_kernel<<<(K * T + 255) / 256, 256, 0, st>>>(static_cast<const uint8_t *>(ids->data), ids->nb[0],
                                                               ids->nb[1], s->ids, K, T);
        // The K-chunked kernel where the shape has a geometry for it and the call more pairs than the small-call limit of
        // the layer entry (there a CTA per item has the shorter latency).  Its map is encoded per call on the host and
        // travels as a launch parameter; a tensor that has none (an odd stride) keeps the kernel chosen above.  Three
        // nodes of 40 pairs ([1536 x 4096] Q2_K twice, [4096 x 1536] Q3_K) with a dense shared expert: 209 -> 162 us.
        CUtensorMap tm;
        PlanBuffers plan = s->plan.b;
        MmidGeom g2;
        const bool v2 = K * T > kSmallCallPairs && mmid_geometry(w->type, I, O, false, &g2, true) == ZMOE_OK && g2.v2 &&
                        (!g2.tiled || make_chunk_map(&tm, w->data, E, O, (int)row, w->nb[2], g2.pitch) == ZMOE_OK);
        if (v2) {
            g = g2;
            plan.mt_gu = plan.mt_dn = g2.maxtok;
        }
        const int nrt = (O + g.R - 1) / g.R;
        if (!rc) rc = launch_plan_from_ids(s->ids, K * T, E, plan, nrt, nrt, st);
        // inactive and out-of-range routes: zero / NaN rows (reference kernels/quant/kquant_matmul.cu:659-662)
        if (!rc) rc = ok(cudaMemsetAsync(y->data, 0, (size_t)T * y->nb[2], st));
        MmidLaunch m;
        m.type = w->type; m.dual = false;
        m.w0 = w->data; m.w1 = nullptr;
        m.stride0 = w->nb[2]; m.stride1 = 0;
        m.total0 = (size_t)(E - 1) * w->nb[2] + (size_t)O * row; m.total1 = 0;
        m.I = I; m.O = O;
        m.q8 = s->q8; m.xdiv = xr == 1 ? K : 1;
        m.y = static_cast<float *>(y->data); m.ldy = (int)(y->nb[1] / 4);
        m.plan = plan; m.down = false;
        if (v2 && g2.tiled) m.tm0 = &tm;
        m.clamp = 0.f; m.clamp_fused = 0;
        m.err = s->err; m.n_sm = s->n_sm;
        m.multi = T > 1;
        if (!rc) rc = launch_mmid(m, g, st);
        if (!rc) fill_bad_rows(m.y, m.ldy, s->ids, K * T, E, O, st);
        g_launches += 5;
        if (rc) return false;
    } else if (w->ne[2] == 1 && w->ne[3] == 1 && x->ne[2] == 1 && x->ne[3] == 1 && x->ne[1] > 0 && x->ne[1] <= 65535 &&
               y->ne[1] == x->ne[1] && x->nb[1] % 4 == 0 && y->nb[1] % 4 == 0) {
        if (reinterpret_cast<size_t>(w->data) & 15) return false;
        if (!execute) return true;
        if (dense_matmul(w->type, static_cast<float *>(y->data), static_cast<const float *>(x->data), (int)(x->nb[1] / 4),
                         w->data, (int)x->ne[1], I, O, (int)(y->nb[1] / 4), st))
            return false;
    } else {
        return false;
    }
    g_hook_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaPeekAtLastError() == cudaSuccess;
}

bool zeromoe_install_f32_quant_graph_hook(void) { return false; }
uint64_t zeromoe_f32_quant_graph_launches(void) { return g_hook_launches.load(std::memory_order_relaxed); }

// ---------------------------------------------------------------------------
// parity hooks
// ---------------------------------------------------------------------------
int zmoe_quantize_q8_K(const float *x_dev, void *blocks_dev, int rows, int I, int for_type, void *stream) {
    if (!x_dev || !blocks_dev || rows <= 0 || I <= 0 || I % QK_K) return ZMOE_ERR_ARG;
    if (block_bytes(for_type) == 0) return ZMOE_ERR_TYPE;
    DeviceScratch *s;
    ScratchLock lock;
    int rc = scratch_get(rows, I, 1, rows, &s, lock);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // quantise into the packed row layout that weight format uses, then regroup into ggml blocks
    const int layout = q8_layout_of(for_type);
    if (!rc) rc = launch_quantize_rows(x_dev, I, s->q8, rows, I, layout, st);
    if (!rc) rc = launch_q8rows_to_blocks(s->q8, static_cast<uint8_t *>(blocks_dev), rows, I, layout, st);
    g_launches += 2;
    return rc;
}

int zmoe_block_isums(int type, const void *w_dev, const float *x_dev, int32_t *isum_dev, int32_t *msum_dev, int rows,
                     int I, void *stream) {
    if (!w_dev || !x_dev || !isum_dev || !msum_dev || rows <= 0 || I <= 0 || I % QK_K) return ZMOE_ERR_ARG;
    if (block_bytes(type) == 0) return ZMOE_ERR_TYPE;
    DeviceScratch *s;
    ScratchLock lock;
    int rc = scratch_get(rows, I, 1, rows, &s, lock);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (!rc) rc = launch_quantize_rows(x_dev, I, s->q8, rows, I, q8_layout_of(type), st);
    if (!rc) rc = launch_block_isums(type, w_dev, s->q8, isum_dev, msum_dev, rows, I, st);
    g_launches += 2;
    return rc;
}

int zmoe_block_isums_pairs(int type, const void *w_dev, const float *x_dev, int32_t *sums_dev, int pairs, int I, void *stream) {
    if (!w_dev || !x_dev || !sums_dev || pairs < 1 || pairs > 4 || I <= 0 || I % QK_K) return ZMOE_ERR_ARG;
    if (block_bytes(type) == 0) return ZMOE_ERR_TYPE;
    DeviceScratch *s;
    ScratchLock lock;
    int rc = scratch_get(pairs, I, 1, pairs, &s, lock);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (!rc) rc = launch_quantize_rows(x_dev, I, s->q8, pairs, I, q8_layout_of(type), st);
    if (!rc) rc = launch_mma_isums(type, w_dev, s->q8, sums_dev, I, pairs, st);
    g_launches += 2;
    return rc;
}

}  // extern "C"

