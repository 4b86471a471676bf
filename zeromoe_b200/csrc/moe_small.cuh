// moe_small.cuh -- a whole MoE layer of very few (token, expert) pairs inside one cooperative kernel: router, top-k, gate / up,
// SwiGLU, down, weighted sum.
//
// Same arithmetic as the five launches it stands for (router_decode_kernel, mmid_kernel twice, quantize_rows_kernel,
// combine_kernel; reference core/moe_router_service.cpp:1409-1474, core/batched_dispatch_pipeline.cpp:1833-1921,
// models/graph/moe_routed_ggml.hpp:198-215).  For one token with up to eight experts the sums also have their order, so that the
// results are theirs bit for bit.
// With a pair or two per expert and a few megabytes of weights those launches were bound by
// their chain: each waits for the one before it to drain, reads its plan, fills its pipeline and drains again.  Here one CTA per SM
// runs through the phases with grid-wide barriers between them (a cooperative launch, so all CTAs are resident):
//   1  the CTA's experts' logits for all tokens; the tokens' rows quantised to Q8_K, by every CTA for itself
//   -- barrier --
//   2  top-k, by every CTA for itself, one warp per token; then gate / up: a warp takes row r of a pair, its bytes copied to shared
//      memory by bulk copies, several rows ahead
//   -- barrier, with the first down rows already on their way --
//   3  the pairs' SwiGLU rows quantised, by every CTA for itself; then down: a warp takes output element d of a token, groups of its lanes
//      multiply the rows d of its K experts side by side, and the weighted sum in k order needs no other warp
// Afterwards the context holds what the separate launches leave there: routes, probabilities, SwiGLU rows, quantised input, plan.
// What other CTAs wrote in the same launch is read past the L1 cache.  Every wait is bounded; on expiry the error flag is raised and
// the CTA goes on without waiting.
#pragma once

#include <type_traits>

#include "mmid.cuh"
#include "q8k.cuh"
#include "zmoe_internal.h"
#define ZMOE_PLAN_ONLY
#include "router.cuh"

namespace zmoe {

constexpr int SMALL_WARPS = 16, SMALL_THREADS = 32 * SMALL_WARPS;
constexpr int SMALL_PAIRS = 32;      // most pairs of a call
constexpr int SMALL_SLOTS = 4;       // most slots of a warp's staging area: rows (pairs of rows, K rows) on their way

// A selection score as an integer that orders like it, 0 for none (a NaN); -0 counts as 0 and -inf is a candidate
__device__ __forceinline__ unsigned score_key(float s) {
    const unsigned u = __float_as_uint(__fadd_rn(s, 0.f));
    return isnan(s) ? 0u : (u >> 31) ? ~u : u | 0x80000000u;
}

// route_token_warp for up to 256 experts in one group, in registers: lane l holds experts l, l + 32, ..  A round is two integer reductions
// over the warp and a new look of one lane at its eight scores.  (In the decode router the same form made the calls slower, 66 -> 70 us
// for a layer of 4096 / 1536 with three tokens, by what it adds to that kernel's code and registers.)
__device__ __forceinline__ void route_token_regs(const RouterSpec &sp, const float *row_in, const float *bias,
                                                 int32_t *ids, float *weights, float *prob_s, int lane) {
    const int E = sp.E, K = sp.K;
    float pr[8];
    unsigned key[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) pr[i] = lane + 32 * i < E ? row_in[lane + 32 * i] : -CUDART_INF_F;
    if (sp.gating == 0) {
        float mx = -CUDART_INF_F;
#pragma unroll
        for (int i = 0; i < 8; ++i) mx = fmaxf(mx, pr[i]);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (lane + 32 * i < E) {
                pr[i] = expf(pr[i] - mx);
                sum += pr[i];
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        const float inv = 1.0f / sum;
#pragma unroll
        for (int i = 0; i < 8; ++i) pr[i] *= inv;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (lane + 32 * i < E) pr[i] = gate_scalar(pr[i], sp.gating);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int e = lane + 32 * i;
        key[i] = 0u;
        if (e < E) {
            prob_s[e] = pr[i];
            key[i] = score_key(pr[i] + (bias ? bias[e] : 0.f));
        }
    }
    __syncwarp();
    // the lane's best, the first on a tie
    unsigned bk;
    int bi;
    auto look = [&]() {
        bk = 0u;
        bi = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (key[i] > bk) { bk = key[i]; bi = i; }
    };
    look();
    float sum_w = 0.f, mine = 0.f;
    int my_id = 0;
    for (int k = 0; k < K; ++k) {
        const unsigned m = __reduce_max_sync(0xffffffffu, bk);
        const unsigned win = m == 0u ? 0u : __reduce_min_sync(0xffffffffu, bk == m ? (unsigned)(lane + 32 * bi) : 0xffffffffu);
        const float w = prob_s[win];
        if (lane == (int)(win & 31u)) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (i == (int)(win >> 5)) key[i] = 0u;      // taken
            look();
        }
        if (lane == k) { mine = w; my_id = (int)win; }
        sum_w += w;
    }
    if (sp.normalize) mine *= 1.0f / fmaxf(sum_w, 6.103515625e-5f);
    if (sp.weight_scale != 0.0f) mine *= sp.weight_scale;
    if (lane < K) {
        ids[lane] = my_id;
        weights[lane] = mine;
    }
}

struct SmallArgs {
    const float *x, *wr, *bias;
    int T, D, F, E, K;
    RouterSpec sp;
    const uint8_t *wg, *wu, *wd;
    size_t sg, su, sd;               // bytes between experts
    int rb_gu, rb_dn;
    float clamp;
    int clamp_fused;
    float *logits;                   // [T, E]; probabilities afterwards
    int32_t *ids;
    float *weights;
    uint8_t *q8x;
    float *act, *out;
    int accumulate;
    PlanOut plan;
    int *err, *bad;
    unsigned *bar;                   // [2] arrivals and departures, zero between launches
    int depth_gu, depth_dn;          // rows (pairs of rows, K rows) a warp has on their way
    int stage;                       // bytes of a warp's staging area
};

struct SmallLaunch;
struct RouterArgs;
SmallArgs small_args(const RouterArgs &r, const SmallLaunch &L);   // all but the staging geometry

// a CTA's shared memory
struct SmallShared {
    uint32_t stage;                  // this warp's staging area
    uint64_t *bars;                  // [SMALL_SLOTS] this warp's: the rows of a slot of the area have landed
    uint32_t phase;                  // the slots' next phases, a bit each
    int *late;                       // set where a wait ran out
    uint8_t *q8x, *q8f;              // packed rows of the input [T] and of the SwiGLU output [T * K]
    float *prob;                     // probabilities and selection scores, 2 E floats per token
    int *ids;                        // [SMALL_PAIRS]
    float *w;                        // [SMALL_PAIRS]
    float *part;                     // [SMALL_WARPS]
};

// grid-wide barrier number `n` (1, 2, ...) of a cooperative launch; expired() is called by one thread if the wait runs out
template <typename Expired>
__device__ __forceinline__ void small_grid_barrier(unsigned *bar, unsigned n, Expired expired) {
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        const unsigned want = n * gridDim.x;
        bool ok = false;
        for (unsigned i = 0; i < (1u << 20) && !ok; ++i) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            ok = v >= want;
        }
        if (!ok) expired();
    }
    __syncthreads();
}
// the last CTA to leave resets the counters for the next launch
__device__ __forceinline__ void small_leave(unsigned *bar) {
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(bar + 1, 1u) == gridDim.x - 1) {
            bar[0] = 0u;
            bar[1] = 0u;
        }
    }
}

// `bytes` bytes at byte `at` of a tensor go to dst, keeping their offset from a 16-byte boundary; called by one lane.
// dst has room for bytes + 32.  Only whole 16-byte pieces are read, all of them the tensor's: it begins and ends on a 16-byte boundary, since
// a matrix has a multiple of 256 rows, or (the QKV matrix and the output head) rows of a multiple of 272 bytes.
// One bulk copy per row and not 16 bytes per lane: those wait at the load / store unit for the rows before them, so that a warp multiplied
// its first row only when its last was nearly there, and came to the grid's barrier late by what it had sent for beforehand (a
// layer of 2048 / 768, one token: fetching 4 200 cycles before gate / up, 4 400 before the barrier after it).
__device__ __forceinline__ void small_stage(uint32_t dst, const uint8_t *w, size_t at, int bytes, uint64_t *bar) {
    const int off = (int)(at & 15);
    const uint32_t n = (uint32_t)((off + bytes + 15) & ~15);
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(n) : "memory");
    bulk_g2s_addr(dst, w + (at - off), n, bar);
}
// after a slot's copies have been issued; called by the warp
__device__ __forceinline__ void small_issued(uint64_t *bar, int lane) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}
// a slot's rows have landed
__device__ __forceinline__ void small_wait(SmallShared &s, int slot) {
    if (!mbar_wait(&s.bars[slot], (s.phase >> slot) & 1u)) *s.late = 1;
    s.phase ^= 1u << slot;
    __syncwarp();
}
// The kernel's barriers; called by all threads, before a CTA barrier that orders them before their use
__device__ __forceinline__ void small_init(uint64_t (*bars)[SMALL_SLOTS], int *late) {
    if (threadIdx.x < SMALL_WARPS * SMALL_SLOTS) mbar_init(&bars[0][0] + threadIdx.x, 1);
    if (threadIdx.x == 0) *late = 0;
    mbar_init_fence();
}

__device__ __forceinline__ void small_prefetch_router(const SmallArgs &a) {
    for (int e = blockIdx.x; e < a.E; e += gridDim.x)
        for (int i = threadIdx.x; i < a.D / 32; i += SMALL_THREADS)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(a.wr + (size_t)e * a.D + 32 * i));
}

// Half of the CTA (256 threads) meets on named barrier 1 or 2
__device__ __forceinline__ void small_half_sync(int half) {
    if (half == 0) asm volatile("bar.sync 1, 256;" ::: "memory");
    else asm volatile("bar.sync 2, 256;" ::: "memory");
}

// phase 1.  x: the tokens' rows [T][D], in global or shared memory.  A logit is the work of half of the CTA: 256 threads, whose sums and
// their order are those of router_decode_kernel.
template <int GU>
__device__ __forceinline__ void small_logits(const SmallArgs &a, const SmallShared &s, const float *x) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, D = a.D;
    constexpr int HT = SMALL_THREADS / 2, HW = SMALL_WARPS / 2;
    static_assert(HT == 256, "threads per logit of router_decode_kernel");
    const int half = tid / HT, ht = tid % HT;
    const int n = (a.E - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x * a.T;   // logits of this CTA's experts, none past the last
    for (int i = half; i < n; i += 2) {
        const int e = (int)blockIdx.x + i / a.T * (int)gridDim.x, t = i % a.T;
        const float4 *wr = reinterpret_cast<const float4 *>(a.wr + (size_t)e * D);
        const float4 *xr = reinterpret_cast<const float4 *>(x + (size_t)t * D);
        float v = 0.f;
        for (int d0 = ht; d0 < D / 4; d0 += 2 * HT) {       // the loads of two steps at once (of four: 0.5 us more per layer of a decoder step)
            float4 w[2], u[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int d = d0 + k * HT;
                w[k] = d < D / 4 ? __ldg(wr + d) : make_float4(0.f, 0.f, 0.f, 0.f);
                u[k] = d < D / 4 ? xr[d] : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                v = fmaf(w[k].x, u[k].x, v); v = fmaf(w[k].y, u[k].y, v); v = fmaf(w[k].z, u[k].z, v); v = fmaf(w[k].w, u[k].w, v);
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (lane == 0) s.part[warp] = v;
        small_half_sync(half);
        if (ht == 0) {
            float sum = 0.f;
#pragma unroll
            for (int w = 0; w < HW; ++w) sum += s.part[HW * half + w];
            a.logits[(size_t)t * a.E + e] = sum;
        }
        if (i + 2 < n) small_half_sync(half);
    }
    const int nb = D / QK_K, str = q8row_stride(D);
    for (int i = warp; i < a.T * nb; i += SMALL_WARPS)
        quantize_block_q8k<false, true>(x + (size_t)(i / nb) * D + QK_K * (i % nb), s.q8x + (i / nb) * str, D, i % nb, lane, q8_layout_of(GU));
}

// A unit's share of a row's sum.  ONE: in f32.  Otherwise the four units of a super-block, on lanes 4i to 4i + 3, meet as integers first
// and all four lanes add the same share: with a rounding per unit the rows of several tokens were further from 64 bits than those of
// the kernels that take such calls otherwise (SwiGLU rows of Q2_K, 2048 / 768: 1.20e-7 of their size against 1.06e-7, this way 1.03e-7).
template <int TYPE, bool ONE>
__device__ __forceinline__ void small_add(float &v, int is, int ms, float d, float dm, float dx, bool on) {
    if (!ONE) {
        is += __shfl_xor_sync(0xffffffffu, is, 1);
        is += __shfl_xor_sync(0xffffffffu, is, 2);
        if (QTraits<TYPE>::kHasMin) {
            ms += __shfl_xor_sync(0xffffffffu, ms, 1);
            ms += __shfl_xor_sync(0xffffffffu, ms, 2);
        }
    }
    if (on) {
        v = fmaf(d * dx, (float)is, v);
        if (QTraits<TYPE>::kHasMin) v = fmaf(-(dm * dx), (float)ms, v);
    }
}

// phase 2: routes, then SwiGLU(gate, up) of the warp's rows into a.act
template <int GU, SmallSums SUMS>
__device__ __forceinline__ void small_gate_up(const SmallArgs &a, SmallShared &s) {
    constexpr bool ONE = SUMS != SUMS_BLOCKS, SHORT = SUMS == SUMS_SHORT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, D = a.D, F = a.F, E = a.E, K = a.K;
    if (warp < a.T) {
        float *const prob = s.prob + 2 * E * warp, *const sel = prob + E;
        for (int e = lane; e < E; e += 32) sel[e] = __ldcg(a.logits + (size_t)warp * E + e);
        __syncwarp();
        route_token_regs(a.sp, sel, a.bias, s.ids + warp * K, s.w + warp * K, prob, lane);
    }
    __syncthreads();
    const int gw = blockIdx.x * SMALL_WARPS + warp, W = gridDim.x * SMALL_WARPS;
    const int n_units = a.T * K * F, room = (a.rb_gu + 47) & ~15, str = q8row_stride(D), U = D / 64;
    // unit u is row u % F of pair u / F; the next of the warp's units to fetch and the one at hand move on by W, without divisions
    const int step_p = W / F, step_r = W - step_p * F;
    int fu = gw, fp = gw / F, fr = gw - fp * F, p = fp, r = fr;
    auto move_on = [&](int &pair, int &row) {
        pair += step_p;
        row += step_r;
        if (row >= F) { row -= F; ++pair; }
    };
    auto fetch = [&](int slot) {
        if (fu < n_units) {
            if (lane < 2)                                // one lane a matrix
                small_stage(s.stage + (uint32_t)((2 * slot + lane) * room), lane ? a.wu : a.wg,
                            (size_t)(uint32_t)s.ids[fp] * (lane ? a.su : a.sg) + (size_t)(uint32_t)fr * (uint32_t)a.rb_gu, a.rb_gu, &s.bars[slot]);
            small_issued(&s.bars[slot], lane);
        }
        fu += W;
        move_on(fp, fr);
    };
#pragma unroll 1
    for (int i = 0; i < a.depth_gu; ++i) fetch(i);
    UnitAct mine;                                          // one token: the lane's unit of its row, for all weight rows
    mine.d = 0.f;
    if (ONE && (SHORT || U <= 32) && lane < U) load_unit_act<GU>(smem_u32(s.q8x), D, lane, mine);
    float keep_g = 0.f, keep_u = 0.f;
    const int keeper = ONE && (SHORT || U <= 32) ? (U - 1) & ~7 : 0;   // first of the eight lanes
    int n_done = 0, slot = 0;
    for (int u = gw; u < n_units; u += W, ++n_done) {
        small_wait(s, slot);
        const uint32_t off = ((uint32_t)r * (uint32_t)a.rb_gu) & 15u;    // experts lie a multiple of 16 bytes apart
        const uint32_t bg = s.stage + (uint32_t)(2 * slot * room) + off, bu = s.stage + (uint32_t)((2 * slot + 1) * room) + off;
        const uint32_t row = smem_u32(s.q8x) + (uint32_t)(ONE ? 0 : (p / K) * str);
        float g = 0.f, v = 0.f;
        if (SHORT || (ONE && U <= 32)) {
            // A unit per lane, added up as by the eight lanes that mmid_kernel gives a row: lane l of eight takes units l, l + 8, .. in turn.
            // The running sums move up eight lanes at a time, so that the last group of eight ends with them.
            int is[2] = {0, 0}, ms[2] = {0, 0};
            float d[2] = {0.f, 0.f}, dm[2] = {0.f, 0.f};
            if (lane < U) {
                unit_dot<GU>(bg + (uint32_t)((lane >> 2) * QTraits<GU>::kBytes), lane & 3, mine, Iq2Tables(), is[0], ms[0], d[0], dm[0]);
                unit_dot<GU>(bu + (uint32_t)((lane >> 2) * QTraits<GU>::kBytes), lane & 3, mine, Iq2Tables(), is[1], ms[1], d[1], dm[1]);
            }
            const float dg = d[0] * mine.d, du = d[1] * mine.d, ig = (float)is[0], iu = (float)is[1];
            const float mg = -(dm[0] * mine.d), mu = -(dm[1] * mine.d), sg = (float)ms[0], su = (float)ms[1];
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                if (n > 0) {
                    if (8 * n >= U) break;
                    g = __shfl_up_sync(0xffffffffu, g, 8);
                    v = __shfl_up_sync(0xffffffffu, v, 8);
                }
                g = fmaf(dg, ig, g);
                v = fmaf(du, iu, v);
                if (QTraits<GU>::kHasMin) {
                    g = fmaf(mg, sg, g);
                    v = fmaf(mu, su, v);
                }
            }
#pragma unroll
            for (int off = 4; off > 0; off >>= 1) {
                g += __shfl_xor_sync(0xffffffffu, g, off);
                v += __shfl_xor_sync(0xffffffffu, v, off);
            }
        } else {
            for (int k0 = 0; k0 < U; k0 += 32) {
                const int k = k0 + lane;
                UnitAct ua;
                int is[2] = {0, 0}, ms[2] = {0, 0};
                float d[2] = {0.f, 0.f}, dm[2] = {0.f, 0.f};
                ua.d = 0.f;
                if (k < U) {
                    load_unit_act<GU>(row, D, k, ua);
                    unit_dot<GU>(bg + (uint32_t)((k >> 2) * QTraits<GU>::kBytes), k & 3, ua, Iq2Tables(), is[0], ms[0], d[0], dm[0]);
                    unit_dot<GU>(bu + (uint32_t)((k >> 2) * QTraits<GU>::kBytes), k & 3, ua, Iq2Tables(), is[1], ms[1], d[1], dm[1]);
                }
                small_add<GU, ONE>(g, is[0], ms[0], d[0], dm[0], ua.d, k < U);
                small_add<GU, ONE>(v, is[1], ms[1], d[1], dm[1], ua.d, k < U);
            }
#pragma unroll
            for (int off = 16; off >= (ONE ? 1 : 4); off >>= 1) {
                g += __shfl_xor_sync(0xffffffffu, g, off);
                v += __shfl_xor_sync(0xffffffffu, v, off);
            }
        }
        // lane i of the eight that hold the sums keeps the i-th row's: SwiGLU runs once for all rows (once per 8)
        if (lane == keeper + (n_done & 7)) { keep_g = g; keep_u = v; }
        __syncwarp();
        fetch(slot);
        slot = slot + 1 == a.depth_gu ? 0 : slot + 1;
        move_on(p, r);
        if (u + W >= n_units || (n_done & 7) == 7) {
            const int nth = lane - keeper, at = u + (nth - (n_done & 7)) * W;
            if (nth >= 0 && nth <= (n_done & 7)) {
                count_bad(a.bad, keep_g, keep_u);
                a.act[at] = swiglu_f(keep_g, keep_u, a.clamp, a.clamp_fused);     // unit u is element u of [T * K][F]
            }
        }
    }
}

// the first down rows of the warp on their way (before the barrier that completes a.act).  ONE: one token
template <bool ONE>
__device__ __forceinline__ void small_fetch_down(const SmallArgs &a, const SmallShared &s, int u, int slot) {
    const int D = a.D, K = a.K, room = (a.rb_dn + 47) & ~15, lane = threadIdx.x & 31;
    if (u < a.T * D) {
        const int t = ONE ? 0 : u / D, d = u - t * D;
        if (lane < K)                                    // one lane a row (K is at most 32)
            small_stage(s.stage + (uint32_t)((slot * K + lane) * room), a.wd,
                        (size_t)(uint32_t)s.ids[t * K + lane] * a.sd + (size_t)(uint32_t)d * (uint32_t)a.rb_dn, a.rb_dn, &s.bars[slot]);
        small_issued(&s.bars[slot], lane);
    }
}
template <bool ONE>
__device__ __forceinline__ void small_prefetch_down(const SmallArgs &a, const SmallShared &s) {
    const int gw = blockIdx.x * SMALL_WARPS + (threadIdx.x >> 5), W = gridDim.x * SMALL_WARPS;
#pragma unroll 1
    for (int i = 0; i < a.depth_dn; ++i) small_fetch_down<ONE>(a, s, gw + i * W, i);
}

// phase 3 (after small_prefetch_down and the barrier)
template <int DN, SmallSums SUMS>
__device__ __forceinline__ void small_down(const SmallArgs &a, SmallShared &s) {
    constexpr bool ONE = SUMS != SUMS_BLOCKS, SHORT = SUMS == SUMS_SHORT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, D = a.D, F = a.F, K = a.K, P = a.T * K;
    const int nb = F / QK_K, str = q8row_stride(F), U = F / 64, room = (a.rb_dn + 47) & ~15;
    for (int i = warp; i < P * nb; i += SMALL_WARPS)
        quantize_block_q8k<true>(a.act + (size_t)(i / nb) * F + QK_K * (i % nb), s.q8f + (i / nb) * str, F, i % nb, lane, q8_layout_of(DN));
    __syncthreads();
    const int gw = blockIdx.x * SMALL_WARPS + warp, W = gridDim.x * SMALL_WARPS;
    int slot = 0;
    for (int u = gw; u < a.T * D; u += W) {
        small_wait(s, slot);
        const int t = ONE ? 0 : u / D, d = u - t * D;
        const uint32_t off = ((uint32_t)d * (uint32_t)a.rb_dn) & 15u;    // experts lie a multiple of 16 bytes apart
        float acc = 0.f;
        // separately rounded products and sums in k order, from the sums of rows k0, k0 + 1, .. in every LPR-th lane
        auto add = [&](int k0, float v, auto lanes) {
            constexpr int LPR = decltype(lanes)::value;
#pragma unroll
            for (int j = 0; j < 32 / LPR; ++j) {
                const float vj = __shfl_sync(0xffffffffu, v, LPR * j);
                if (k0 + j < K) {
                    const float pr = __fmul_rn(s.w[t * K + k0 + j], vj);
                    acc = k0 + j == 0 ? pr : __fadd_rn(acc, pr);
                }
            }
        };
        auto row_of = [&](int k, uint32_t &blk, uint32_t &row) {
            const int p = t * K + k;
            blk = s.stage + (uint32_t)((slot * K + k) * room) + off;
            row = smem_u32(s.q8f) + (uint32_t)(p * str);
        };
        // lanes per row: eight, four rows at once, or the whole warp for rows of more than 32 units
        auto rows = [&](auto lanes) {
            constexpr int LPR = decltype(lanes)::value, NR = 32 / LPR;
            for (int k0 = 0; k0 < K; k0 += NR) {
                const int k = k0 + lane / LPR;
                float v = 0.f;
                uint32_t blk, row;
                row_of(min(k, K - 1), blk, row);
#pragma unroll 1
                for (int i0 = 0; i0 < U; i0 += LPR) {
                    const int i = i0 + lane % LPR;
                    const bool on = k < K && i < U;
                    UnitAct ua;
                    int is = 0, ms = 0;
                    float dw = 0.f, dm = 0.f;
                    ua.d = 0.f;
                    if (on) {
                        load_unit_act<DN>(row, F, i, ua);
                        unit_dot<DN>(blk + (uint32_t)((i >> 2) * QTraits<DN>::kBytes), i & 3, ua, Iq2Tables(), is, ms, dw, dm);
                    }
                    small_add<DN, ONE>(v, is, ms, dw, dm, ua.d, on);
                }
#pragma unroll
                for (int off = LPR / 2; off >= (ONE ? 1 : 4); off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
                add(k0, v, lanes);
            }
        };
        if (!SHORT && U > 32) {
            rows(std::integral_constant<int, 32>());
        } else if constexpr (!ONE) {
            rows(std::integral_constant<int, 8>());
        } else {
            // Four lanes to a row, eight rows at once (K is at most that).  Lane l takes the units of lanes l and l + 4 of the eight that mmid_kernel
            // gives a row, in turn, and keeps their sums apart.
            float v0 = 0.f, v1 = 0.f;
            if (lane >> 2 < K) {
                uint32_t blk, row;
                row_of(lane >> 2, blk, row);
#pragma unroll 1
                for (int i = lane & 3; i < U; i += 4) {
                    UnitAct ua;
                    load_unit_act<DN>(row, F, i, ua);
                    int is, ms;
                    float dw, dm;
                    unit_dot<DN>(blk + (uint32_t)((i >> 2) * QTraits<DN>::kBytes), i & 3, ua, Iq2Tables(), is, ms, dw, dm);
                    v0 = fmaf(dw * ua.d, (float)is, v0);
                    if (QTraits<DN>::kHasMin) v0 = fmaf(-(dm * ua.d), (float)ms, v0);
                    const float next = v1;
                    v1 = v0;
                    v0 = next;
                }
            }
            v0 += v1;
            v0 += __shfl_xor_sync(0xffffffffu, v0, 2);
            v0 += __shfl_xor_sync(0xffffffffu, v0, 1);
            add(0, v0, std::integral_constant<int, 4>());
        }
        if (lane == 0) a.out[u] = a.accumulate ? __fadd_rn(__ldcg(a.out + u), acc) : acc;
        __syncwarp();
        small_fetch_down<ONE>(a, s, u + a.depth_dn * W, slot);
        slot = slot + 1 == a.depth_dn ? 0 : slot + 1;
    }
}

// what the separate launches leave in the context; called by all threads of one CTA, after the second barrier
__device__ __forceinline__ void small_leave_state(const SmallArgs &a, const SmallShared &s) {
    const int tid = threadIdx.x, E = a.E, P = a.T * a.K;
    for (int i = tid; i < a.T * q8row_stride(a.D) / 16; i += SMALL_THREADS)
        reinterpret_cast<uint4 *>(a.q8x)[i] = reinterpret_cast<const uint4 *>(s.q8x)[i];
    for (int i = tid; i < a.T * E; i += SMALL_THREADS) a.logits[i] = s.prob[2 * E * (i / E) + i % E];
    for (int i = tid; i < P; i += SMALL_THREADS) { a.ids[i] = s.ids[i]; a.weights[i] = s.w[i]; }
    __syncthreads();
    int *const cnt = reinterpret_cast<int *>(s.prob);
    build_plan_cta<PLAN_ONE_RUN>(s.ids, P, E, a.plan, cnt, cnt + E + 1, nullptr, nullptr, 1);
    __syncthreads();
}

// GU, DN: Q2_K, Q3_K or Q4_K
template <int GU, int DN, SmallSums SUMS>
__global__ void __launch_bounds__(SMALL_THREADS, 1) moe_small_kernel(const SmallArgs a) {
    // a staging area per warp | packed input rows | packed SwiGLU rows | probabilities and scores
    extern __shared__ __align__(128) uint8_t dyn[];
    __shared__ float s_part[SMALL_WARPS], s_w[SMALL_PAIRS];
    __shared__ int s_ids[SMALL_PAIRS], s_late;
    __shared__ __align__(8) uint64_t s_bars[SMALL_WARPS][SMALL_SLOTS];
    SmallShared s;
    s.bars = s_bars[threadIdx.x >> 5]; s.phase = 0; s.late = &s_late;
    small_init(s_bars, &s_late);                         // used after the first barrier
    s.stage = smem_u32(dyn) + (uint32_t)((threadIdx.x >> 5) * a.stage);
    s.q8x = dyn + SMALL_WARPS * a.stage;
    s.q8f = s.q8x + a.T * q8row_stride(a.D);
    s.prob = reinterpret_cast<float *>(s.q8f + a.T * a.K * q8row_stride(a.F));
    s.ids = s_ids; s.w = s_w; s.part = s_part;
    small_prefetch_router(a);
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    small_logits<GU>(a, s, a.x);
    auto expired = [&]() { atomicExch(a.err, 21); };
    small_grid_barrier(a.bar, 1, expired);
    small_gate_up<GU, SUMS>(a, s);
    small_prefetch_down<SUMS != SUMS_BLOCKS>(a, s);
    small_grid_barrier(a.bar, 2, expired);
    small_down<DN, SUMS>(a, s);
    if (blockIdx.x == gridDim.x - 1) {
        __syncthreads();
        small_leave_state(a, s);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_late) expired();
    small_leave(a.bar);
}

}  // namespace zmoe
