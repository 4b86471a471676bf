// zmoe_internal.h -- host-side declarations shared by the .cu files of the
// library (not part of the public C ABI; see include/zmoe_b200.h for that).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "../../include/zmoe_b200.h"

namespace zmoe {

// ---- small host services shared by the .cu files (implemented in api.cu) ----
// multiprocessor count of the current device (cached per device); 0 on failure
int device_sm_count();
// adds to the counter behind zmoe_kernel_launches()
void count_launches(uint64_t n);
// what zmoe_last_status() returns on this thread
void set_last_status(int rc);
// raises a kernel's dynamic shared-memory limit to at least `bytes` on the current device (the attribute
// is per function and per device; remembered under a mutex)
int raise_dynamic_smem(const void *fn, size_t bytes);
// error word of the no-allocation entry point on the current device, read and cleared; 0 when that entry
// point has not run on this device (implemented in noalloc.cu)
int noalloc_take_error(int *out);

// accessors of the opaque handles for the other .cu files (implemented in api.cu)
// device pointers of the route table a layer's context currently holds, and the layer's expert count
int layer_route_table(zmoe_layer *layer, const int32_t **ids_dev, const float **weights_dev, int *n_experts);
zmoe_ctx *layer_context(zmoe_layer *layer);
// out (+)= MoE(x) for T tokens: the router and the experts in one kernel where the call is small enough, else zmoe_route and zmoe_expert_ffn
int layer_forward(zmoe_layer *layer, const float *x_dev, float *out_dev, int T, int accumulate, void *stream);
int context_path(const zmoe_ctx *ctx);

// device-resident routing plan buffers
struct PlanBuffers {
    int *hdr = nullptr, *active = nullptr, *offs = nullptr, *slot = nullptr;
    int *item_offs_gu = nullptr, *item_offs_dn = nullptr, *freq = nullptr;
    int *aoffs = nullptr, *antok = nullptr;
    int *pos = nullptr;    // [P] position of each pair in expert order (inverse of slot), -1 = inactive; optional
    int cap_e = 0;
    int mt_gu = 4, mt_dn = 4;   // pairs per item of the two projections (the geometry's maxtok)
};

constexpr int ROUTER_MAX_GROUPS = 64;   // token groups (of 4) the decode router can ticket: 256 tokens

struct RouterArgs {
    const float *x;        // [T, D]
    const float *wr;       // [E, D]
    const float *bias;     // [E] or null
    int T, D, E, K;
    int gating, normalize;
    float weight_scale;
    int n_groups, n_groups_used;
    float *logits;         // [T, E] scratch; holds probabilities afterwards
    int32_t *ids;          // [T, K]
    float *weights;        // [T, K]
    uint8_t *q8x;          // packed Q8_K rows of x, [T, q8row_stride(D)]
    int q8_layout;         // unit layout of q8x (that of the gate / up weight format)
    PlanBuffers plan;
    int nrt_gu, nrt_dn;
    unsigned *ticket;      // 1 + ROUTER_MAX_GROUPS zero-initialised counters, left at zero
    bool want_q8x = true;  // large batches: also quantise x into q8x (the tensor-core path does not read it)
    float *logits_part = nullptr;  // large batches: [ksplit][T, E] partial logits of a k-split router GEMM, or null
    long logits_part_rows = 0;     // rows of E it holds: ksplit * T stays within them
    int n_sm = 0;
    unsigned long long *stats = nullptr;   // phase timers of the decode router (builds with ZMOE_GEMM_STATS), or null
};
constexpr int ROUTER_MAX_SPLIT = 16;
// The tiled router or the decode router.  The decode router's CTA per (expert, 4 tokens) reads every activation row E times, so it
// grows with T * E; the tiles split k up to sixteen ways, so they take as long as D / 16 products and three more launches whatever
// the batch is.  A route call, decode against tiled, us: hidden 2048, 128 experts: 97 tokens 30 / 24, 256 61 / 27; 7168, 256
// experts: 97 66 / 44, 256 150 / 66; 4096, 64 experts: 97 23 / 27, 128 27 / 28, 256 43 / 27; 7168, 64 experts: 97 26 / 36,
// 160 37 / 37; 4096, 32 experts: 160 22 / 24, 256 29 / 25; 4096, 8 experts: 256 18 / 24.  Both have the same short sums up to
// ROUTER_SHORT_TOKENS; larger batches take the tiles alone, with longer ones.
constexpr int ROUTER_TILED_TOKENS = 96, ROUTER_SHORT_TOKENS = 256;
constexpr int ROUTER_TILED_EXPERTS = 1536;   // the tiled router's selection holds this many in shared memory
constexpr int ROUTER_DECODE_HIDDEN = 8192;   // the decode router holds a row of this many elements in registers
inline bool router_takes_tiles(long T, long D, long E) {
    if (T > ROUTER_SHORT_TOKENS) return true;
    if (T <= ROUTER_TILED_TOKENS || E > ROUTER_TILED_EXPERTS) return false;
    return 5 * T * E > 8 * D || D > ROUTER_DECODE_HIDDEN;
}
inline long router_part_rows(long max_tokens) {
    const long split = ROUTER_MAX_SPLIT * (max_tokens < 1024 ? max_tokens : 1024);
    return split > 4 * max_tokens ? split : 4 * max_tokens;
}

// geometry of one mmid launch, fixed per (type, I, O)
struct MmidGeom {
    int lpr, upl, ncw;     // lanes per row, units per lane, consumer warps
    int R;                 // rows per tile
    int nstage, stage_bytes, wtile_bytes;
    int rbs, q8s;          // shared-memory strides of weight rows and of activation rows
    size_t smem_bytes;
    // K-chunked kernel (mmid2.cuh), chosen where the shape allows it and the caller can supply its maps
    int v2 = 0;            // 1: launch_mmid takes the K-chunked kernel; R is then 32
    int cb = 0, nch = 0;   // super-blocks per chunk, chunks per row
    int acb = 0;           // super-blocks of the activation slice a stage holds (cb, or 4 where cb is 2)
    int pitch = 0;         // bytes between rows of a chunk in shared memory
    int lb_log2 = 0;       // log2 of the lanes that share a row on the one-pair path
    int q8s_l = 0;         // bytes between the pairs' activation slices in shared memory
    int maxtok = 4;        // pairs per item (8 where the K-chunked kernel has the tensor-core path and the stages fit)
    int tiled = 0;         // chunks come through tiled maps (make_chunk_map); 0: rows are copied whole as one run
    // tensor-core kernel (mmid_tc.cuh): tc_geometry fills these, R (rows of one matrix per item) and pitch
    int tc = 0, g_log2 = 0, cb_log2 = 0;
};
// allow_v2: the caller passes maps made by make_chunk_map where g->tiled is set
int mmid_geometry(int type, int I, int O, bool dual, MmidGeom *g, bool allow_v2 = false);
// whether the kernel of a geometry that is not the K-chunked one reads a weight row once for several pairs of an expert
bool mmid_shares_rows(int type, const MmidGeom &g, int I, bool dual);
// Map of a [E][O rows][rb bytes] weight tensor whose box is 32 rows of `pitch` bytes starting at any multiple of 16
// bytes inside a row: bytes past the end of a row and rows past the last arrive as zeros.
int make_chunk_map(CUtensorMap *m, const void *base, int E, int O, int rb, size_t expert_stride, int pitch);

// Geometry of the integer tensor-core kernel for experts that hold several pairs; its maps come from make_tc_map.
int tc_geometry(int type, int I, int O, bool dual, MmidGeom *g);
// most pairs per item of that kernel, for calls of T tokens: what a call's plan is built with
int tc_maxtok(int T);
// Map of a [E][O rows][rb bytes] weight tensor, G = 2^g_log2 rows at a time (G * rb a multiple of 16): box of 64 / G groups x `pitch` bytes
int make_tc_map(CUtensorMap *m, const void *base, int E, int O, int rb, size_t expert_stride, int pitch, int g_log2);

struct MmidLaunch {
    int type;
    bool dual;
    const void *w0, *w1;
    size_t stride0, stride1, total0, total1;
    int I, O;
    const uint8_t *q8;
    int xdiv;
    float *y;
    int ldy;
    PlanBuffers plan;
    bool down;             // use the down-projection item space
    float clamp;
    int clamp_fused;
    int *err;
    int *bad = nullptr;    // [2] NaN / Inf counters of the fused SwiGLU epilogue, or null
    int *queue = nullptr;  // [4] zeroed ints: the chunked kernel deals its items through a ticket counter (two ints per
                           // projection, left zero by every launch); null = items dealt round-robin over the grid
    int n_sm;
    bool multi = false;    // some expert may hold two or more pairs: allow the tensor-core consumer path
    // optional tiled maps of w0 / w1 (make_rows_map) that deliver tiles with padded rows in one copy
    const CUtensorMap *tm0 = nullptr, *tm1 = nullptr;
};
// Map of a [E][O rows][rb bytes] weight tensor whose box is R rows of rb + 16 bytes: the 16 bytes past the
// end of a row are out of bounds and arrive as zeros, which pads the rows in shared memory.  Rows up to 2032 bytes.
int make_rows_map(CUtensorMap *m, const void *base, int E, int O, int rb, size_t expert_stride, int R);
// dst[i] = (float)src[i] for n bf16 values (n a multiple of 8, both 16-byte aligned)
int launch_widen_bf16(const void *src, float *dst, long n, int n_sm, cudaStream_t st);
// g[t] = sigmoid(w . x[t]) for T rows of D floats (D a multiple of 4)
int launch_token_gate(const float *x, const float *w, float *g, int T, int D, cudaStream_t st);
int launch_mmid(const MmidLaunch &L, const MmidGeom &g, cudaStream_t st);
int launch_mmid_tc(const MmidLaunch &L, const MmidGeom &g, cudaStream_t st);
// s32 sums of the tensor-core consumer path: out[16 rows][4 pair slots][I / 256][2]
int launch_mma_isums(int type, const void *w, const uint8_t *q8, int *out, int I, int pairs, cudaStream_t st);

// prefill path: tcgen05 grouped GEMM over fp16 activations (Q8_K round trip applied, rows scaled)
struct GemmLaunch {
    int type;
    bool dual;
    const void *w0, *w1;
    size_t stride0, stride1;
    int n_experts;         // experts the weight tensors hold
    int I, O;
    const void *x_f16;     // sorted activation rows [x_rows, I] fp16
    const float *xscale;   // their per-row scales
    int x_rows;            // rows the buffer holds
    float *y;
    int ldy;
    PlanBuffers plan;
    float clamp;
    int clamp_fused;
    int *err;
    int *bad = nullptr;    // [2] NaN / Inf counters of the fused SwiGLU epilogue, or null
    int n_sm;
};
bool gemm_sm100_supported(int type, int I, int O);
bool gemm_sm100_built(int type);   // the type's compiled kernels have the registers their roles share out
unsigned long long *gemm_stats_buffer(int which);
int gemm_stats_read(unsigned long long *out32);
int launch_gemm_sm100(const GemmLaunch &L, cudaStream_t st);
int launch_q8_roundtrip_f16(const float *x, int ldx, void *out_f16, float *scale, const PlanBuffers &plan,
                            int max_rows, int xdiv, int I, cudaStream_t st);
// the same for the layer input, where the K pairs of a token share one source row: the row is passed through
// Q8_K once and written to the K positions plan.pos names (needs plan.pos)
int launch_q8_roundtrip_tokens_f16(const float *x, int ldx, void *out_f16, float *scale, const PlanBuffers &plan,
                                   int T, int K, int I, cudaStream_t st);

int launch_router_decode(const RouterArgs &a, cudaStream_t st);
int launch_router_prefill(const RouterArgs &a, cudaStream_t st);  // four launches; for large T
// the planner, first copying routes from outside into the context's tables (ids, w); window: expert numbers
// outside [first, first + E) become -1
int launch_plan_ingest(const int32_t *src_ids, const float *src_w, int32_t *ids, float *w, int P, int E, int first,
                       bool window, const PlanBuffers &plan, int nrt_gu, int nrt_dn, cudaStream_t st, int topk = 0, int ids_ld = 0, int w_ld = 0);
int launch_plan_from_ids(const int32_t *ids, int P, int E, const PlanBuffers &plan, int nrt_gu, int nrt_dn,
                         cudaStream_t st);
int launch_plan_dense(int S, const PlanBuffers &plan, int nrt, cudaStream_t st);
int launch_quantize_rows(const float *x, int ldx, uint8_t *q8, int rows, int I, int layout, cudaStream_t st);
int launch_q8rows_to_blocks(const uint8_t *q8, uint8_t *blocks, int rows, int I, int layout, cudaStream_t st);
int launch_combine(float *out, const float *y, const float *w, const int32_t *ids, int T, int K, int D, int E,
                   int accumulate, cudaStream_t st);
int launch_block_isums(int type, const void *w, const uint8_t *q8, int32_t *isum, int32_t *msum, int rows, int I,
                       cudaStream_t st);

// a whole layer of very few pairs in one cooperative kernel (moe_small.cuh)
struct SmallLaunch {
    int type_gu, type_dn, F;
    const void *w_gate, *w_up, *w_down;
    size_t stride_gate, stride_up, stride_down;
    float clamp;
    int clamp_fused;
    float *act, *out;
    int accumulate;
    int *err, *bad;
    unsigned *bar;         // [2] zero-initialised, left at zero
};
// calls whose separate launches take their pairs one at a time with mmid_kernel
constexpr int kSmallCallPairs = 8;
// How the one-kernel forms add up a row.  One token with at most that many experts: in the order of those launches, rows of up to 2048
// (eight lanes each) or longer ones too; a form for short rows alone because a layer's phases run once each and wait for their
// instructions: 48 layers of 2048 / 768 take 2480 us with it, 2557 with the branches for long rows beside theirs.  Otherwise a super-block's integers first.
enum SmallSums { SUMS_BLOCKS, SUMS_LONG, SUMS_SHORT };
inline SmallSums small_sums(int T, int K, int D, int F) {
    return T > 1 || K > kSmallCallPairs ? SUMS_BLOCKS : D > 2048 || F > 2048 ? SUMS_LONG : SUMS_SHORT;
}
bool moe_small_supported(int gu, int dn, int T, int D, int F, int E, int K);
// ZMOE_ERR_STATE where the device cannot hold the whole grid at once (the caller takes the separate launches)
int launch_moe_small(const RouterArgs &r, const SmallLaunch &L, cudaStream_t st);
// status of a cooperative launch: ZMOE_ERR_STATE, with the error cleared, where it was refused for its size
inline int cooperative_status(cudaError_t e) {
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
        cudaGetLastError();
        return ZMOE_ERR_STATE;
    }
    return e == cudaSuccess ? ZMOE_OK : ZMOE_ERR_CUDA;
}

// router and launch arguments of that kernel for a call of T tokens of a layer; false where the call does not take it.  Whether the
// context's path allows it (0 or 1) is the caller's to see when it launches.  Nothing of the context changes.
bool layer_small_args(zmoe_layer *layer, const float *x_dev, float *out_dev, int T, int accumulate, RouterArgs *r, SmallLaunch *s);
// host state of the layer's context after such a call
void layer_small_done(zmoe_layer *layer, const float *x_dev, int T);

// one token through a decoder in one cooperative kernel (decoder_step.cuh)
struct DecoderStep;
struct DecoderStepDesc {
    int n_layers;
    const float *const *attn_norm, *const *ffn_norm;
    const void *const *wqkv, *const *wo;
    zmoe_layer *const *moe;
    const void *embd, *head;
    const float *out_norm;
    int D, H, KV, HD, vocab, max_ctx, splits;
    float eps, theta_scale, scale;
    float *h, *xn, *qkv, *part, *logits, *ad;
    int8_t *aq;
    void *kc, *vc;
    int *pos;
    int32_t *next;
    unsigned *sync;        // decoder_step_sync_words(KV) zero-initialised words, 8-byte aligned, left at zero
};
int decoder_step_sync_words(int KV);
// null where the decoder's shapes or layers do not allow it
DecoderStep *decoder_step_create(const DecoderStepDesc &d);
void decoder_step_destroy(DecoderStep *s);
// ZMOE_ERR_STATE where a layer's context is set to a path that the kernel does not follow, or the device cannot hold the whole grid at once:
// the caller takes the separate launches
int decoder_step_launch(DecoderStep *s, const int32_t *token_dev, cudaStream_t st);

// launch helper: programmatic dependent launch attribute on every kernel of the chain
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                              Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

}  // namespace zmoe
