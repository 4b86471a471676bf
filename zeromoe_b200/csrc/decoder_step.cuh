// decoder_step.cuh -- one token through the whole decoder in one cooperative kernel: embedding, then per layer norm, QKV projection, RoPE
// and cache, attention, output projection, norm, MoE layer, and at the end norm, output head and arg-max.
//
// Same arithmetic as the launches of decoder.cu it stands for (see there for what each follows in the reference), with every sum in their
// order: with up to eight experts per token its results are theirs bit for bit.  A one-token step
// streams little (a layer of 2048 / 768 about 40 MB) and was bound by its chain of launches, 26 for two layers at 5 to 6 us each.  Here
// one CTA per SM runs through the phases, with six grid-wide barriers per layer (a cooperative launch, so all CTAs are resident);
// whatever a phase needs that does not depend on the one before it -- its warps' first weight rows -- is on its way before the barrier,
// and what is small (norms, quantising a row, top-k) every CTA does for itself instead of waiting for another.
//   barrier 1 after QKV, 2 after attention (the last CTA of a KV head merges its shares and quantises them), 3 after the output
//   projection, 4 after the router's logits, 5 after gate / up, 6 after down
// The residual stream lives in global memory; what other CTAs wrote in the same launch is read past the L1 cache.
#pragma once

#include "moe_small.cuh"

namespace zmoe {

struct StepLayer {
    const float *attn_norm, *ffn_norm;
    const uint8_t *wqkv, *wo;
    SmallArgs moe;            // x unused; out is the residual stream
    int leave_state;          // 1: the last layer that uses its context
};

struct StepArgs {
    const StepLayer *layers;
    int n_layers;
    const int32_t *token;     // device
    const uint8_t *embd, *head;
    const float *out_norm;
    int D, H, KV, HD, vocab, max_ctx;
    float eps, theta_scale, scale;
    float *h, *xn, *qkv, *part, *logits;
    int8_t *aq;               // quantised attention output
    float *ad;
    __half *kc, *vc;          // [layers][max_ctx][KV * HD]
    int *pos;
    int32_t *next;
    unsigned long long *best; // arg-max key, zero between launches
    unsigned *head_ticket;    // [KV] zero between launches
    unsigned *bar;            // [2]
    int splits;               // shares of the keys per KV head
    int stage, depth_q, depth_o;   // bytes of a warp's staging area; rows on their way: rows of D, rows of H * HD
};

// a row of Q8_0 blocks against a quantised activation row, both in shared memory; the arithmetic of q8_0_matmul_kernel
__device__ __forceinline__ float step_row_dot(uint32_t row, const int8_t *aq, const float *ad, int nb, int lane) {
    float acc = 0.f;
    for (int b = lane; b < nb; b += 32) {
        const uint32_t blk = row + 34 * b;
        const float dw = half_bits_to_float(lds16(blk));
        uint32_t qw[8];
        lds32xN_any<2, 8>(blk + 2, qw);
        const uint4 a0 = *reinterpret_cast<const uint4 *>(aq + 32 * b), a1 = *reinterpret_cast<const uint4 *>(aq + 32 * b + 16);
        int sum = __dp4a((int)qw[0], (int)a0.x, 0);
        sum = __dp4a((int)qw[1], (int)a0.y, sum);
        sum = __dp4a((int)qw[2], (int)a0.z, sum);
        sum = __dp4a((int)qw[3], (int)a0.w, sum);
        sum = __dp4a((int)qw[4], (int)a1.x, sum);
        sum = __dp4a((int)qw[5], (int)a1.y, sum);
        sum = __dp4a((int)qw[6], (int)a1.z, sum);
        sum = __dp4a((int)qw[7], (int)a1.w, sum);
        acc = __fadd_rn(acc, __fmul_rn((float)sum, __fmul_rn(dw, ad[b])));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    return acc;
}

// rows gw, gw + W, ... of a Q8_0 matrix, the first `depth` of them on their way (step_prefetch) before the activations are there
__device__ __forceinline__ void step_fetch(const SmallShared &s, const uint8_t *w, int n_rows, int rb, int o, int slot, int lane) {
    if (o >= n_rows) return;
    if (lane == 0) {
        small_stage(s.stage + (uint32_t)(slot * ((rb + 47) & ~15)), w, (size_t)o * rb, rb, &s.bars[slot]);
        mbar_arrive(&s.bars[slot]);
    }
    __syncwarp();
}
__device__ __forceinline__ void step_prefetch(const SmallShared &s, const uint8_t *w, int n_rows, int rb, int depth) {
    const int gw = blockIdx.x * SMALL_WARPS + (threadIdx.x >> 5), W = gridDim.x * SMALL_WARPS;
#pragma unroll 1
    for (int i = 0; i < depth; ++i) step_fetch(s, w, n_rows, rb, gw + i * W, i, threadIdx.x & 31);
}
template <typename Put>
__device__ __forceinline__ void step_rows(SmallShared &s, const uint8_t *w, int n_rows, int rb, int depth, const int8_t *aq, const float *ad, Put put) {
    const int lane = threadIdx.x & 31, gw = blockIdx.x * SMALL_WARPS + (threadIdx.x >> 5), W = gridDim.x * SMALL_WARPS;
    int slot = 0;
    for (int o = gw; o < n_rows; o += W) {
        small_wait(s, slot);
        const float v = step_row_dot(s.stage + (uint32_t)(slot * ((rb + 47) & ~15)) + (uint32_t)(((size_t)o * rb) & 15), aq, ad, rb / 34, lane);
        if (lane == 0) put(o, v);
        __syncwarp();
        step_fetch(s, w, n_rows, rb, o + depth * W, slot, lane);
        slot = slot + 1 == depth ? 0 : slot + 1;
    }
}

// x <- RMSNorm(x) * w, in shared memory, by the whole CTA.  The sum of squares is that of rmsnorm_kernel, by 256 threads in its order.
__device__ __forceinline__ void step_norm(float *x, const float *w, int D, float eps, float *part) {
    constexpr int ST = 256;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid < ST) {
        float ss = 0.f;
        for (int i = tid; i < D / 4; i += ST) {
            const float4 v = reinterpret_cast<float4 *>(x)[i];
            ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) part[warp] = ss;
    }
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < ST / 32; ++i) tot += part[i];
    const float inv = rsqrtf(tot / (float)D + eps);
    for (int i = tid; i < D / 4; i += SMALL_THREADS) {
        const float4 v = reinterpret_cast<const float4 *>(x)[i], g = __ldg(reinterpret_cast<const float4 *>(w) + i);
        reinterpret_cast<float4 *>(x)[i] = make_float4(v.x * inv * g.x, v.y * inv * g.y, v.z * inv * g.z, v.w * inv * g.w);
    }
    __syncthreads();
}
// Q8_0 of x (shared) into q, d (shared), by the whole CTA: a warp per block of 32
__device__ __forceinline__ void step_quantise(const float *x, int8_t *q, float *d, int n) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int b = warp; b < n / 32; b += SMALL_WARPS) {
        const float v = x[32 * b + lane];
        float amax = fabsf(v);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        const float dd = __fdiv_rn(amax, 127.f), id = dd != 0.f ? __fdiv_rn(1.0f, dd) : 0.f;
        q[32 * b + lane] = (int8_t)roundf(__fmul_rn(v, id));
        if (lane == 0) d[b] = __half2float(__float2half_rn(dd));
    }
    __syncthreads();
}

// ---- attention ----
// Keys and values come a chunk of 32 keys at a time, into shared memory, where the heads of a KV head share them.  The chunk that a CTA meets
// first is on its way while the CTA still multiplies rows of the QKV matrix (all of it but the new key lies in the cache since the step
// before), and the dot products and the weighted sum then wait for no trip to memory: with the keys read by every warp for itself, and
// the values eight at a time, attention over 34 to 81 keys took 18 200 cycles per layer, most of it such trips.
constexpr int STEP_KEYS = 32;
__host__ __device__ constexpr int step_kv_pitch(int hd) { return 2 * hd + 16; }      // 128-bit loads of one column meet every bank group
__host__ __device__ constexpr int step_kv_bytes(int hd) { return 2 * STEP_KEYS * step_kv_pitch(hd); }

// the shares of the keys at position p: their number, and the keys of each (a multiple of 32)
__device__ __forceinline__ void step_shares(const StepArgs &a, int p, int &n_keys, int &per, int &ns) {
    n_keys = min(p + 1, a.max_ctx);
    const int chunks = (n_keys + 31) / 32;
    per = (chunks + a.splits - 1) / a.splits;
    ns = (chunks + per - 1) / per;
}
// rows [k0, k0 + 32) of one KV head up to key `end`, without the new one (it is written by the share that holds it); called by all
// warps, which take two keys each (64 copies of one warp kept its rows waiting for 2 800 cycles)
__device__ __forceinline__ void step_fetch_kv(uint32_t kv, const __half *kc, const __half *vc, int KV, int HD, int kvh, int k0, int end, int fresh, uint64_t *bar) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // what was read and written in this memory before, by ordinary loads and stores, comes before the copies
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (threadIdx.x == 0) {
        const int n = max(0, min(STEP_KEYS, end - k0)) - (fresh >= k0 && fresh < min(end, k0 + STEP_KEYS) ? 1 : 0);
        mbar_arrive_expect_tx(bar, (uint32_t)(4 * HD * n));
    }
    const int row = 2 * warp + (lane >> 1), key = k0 + row;
    if (lane < 4 && key < end && key != fresh) {
        const uint32_t dst = kv + (uint32_t)((row + (lane & 1) * STEP_KEYS) * step_kv_pitch(HD));
        bulk_g2s_addr(dst, (lane & 1 ? vc : kc) + ((size_t)key * KV + kvh) * HD, (uint32_t)(2 * HD), bar);
    }
    __syncwarp();
}
static_assert(2 * SMALL_WARPS == STEP_KEYS, "keys of a warp");

// Share z of a KV head's keys: attention_kernel with the rotation of q and of the new key folded in.  qs: [G][HD] shared; kv: the chunk;
// ready: its first chunk is on its way already.  phase: of kv_bar, moved on with every chunk.  False: a wait ran out.
template <int HD>
__device__ __forceinline__ bool step_attention(const StepArgs &a, __half *kc, __half *vc, int kvh, int z, int p, float *qs, const float2 *rot, uint8_t *kv,
                                               uint64_t *kv_bar, uint32_t &phase, bool ready) {
    constexpr int DPL = HD / 32, PITCH = step_kv_pitch(HD);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x, G = a.H / a.KV, KV = a.KV;
    int n_keys, per, ns;
    step_shares(a, p, n_keys, per, ns);
    const int key_lo = min(n_keys, z * per * 32), key_hi = min(n_keys, (z + 1) * per * 32);
    const bool turn = p < a.max_ctx;                     // past the context nothing is rotated or appended
    const bool fresh_here = turn && p >= key_lo && p < key_hi;
    for (int i = tid; i < G * (HD / 2); i += SMALL_THREADS) {
        const int g = i / (HD / 2), j = i % (HD / 2);
        const float2 v = __ldcg(reinterpret_cast<const float2 *>(a.qkv + (size_t)(kvh * G + g) * HD) + j), r = rot[j];
        qs[g * HD + 2 * j] = turn ? __fsub_rn(__fmul_rn(v.x, r.x), __fmul_rn(v.y, r.y)) : v.x;
        qs[g * HD + 2 * j + 1] = turn ? __fadd_rn(__fmul_rn(v.x, r.y), __fmul_rn(v.y, r.x)) : v.y;
    }
    // the new key's halves, by threads whose warps have no head's rotation to wait for
    __half2 fk = __half2half2(__ushort_as_half(0)), fv = fk;
    const int ft = SMALL_THREADS - 1 - tid;
    if (fresh_here && ft < HD / 2) {
        const size_t at = ((size_t)p * KV + kvh) * HD + 2 * ft;
        const float2 k = __ldcg(reinterpret_cast<const float2 *>(a.qkv + (size_t)(a.H + kvh) * HD) + ft), r = rot[ft];
        const float2 v = __ldcg(reinterpret_cast<const float2 *>(a.qkv + (size_t)(a.H + KV + kvh) * HD) + ft);
        fk = __halves2half2(__float2half_rn(__fsub_rn(__fmul_rn(k.x, r.x), __fmul_rn(k.y, r.y))),
                            __float2half_rn(__fadd_rn(__fmul_rn(k.x, r.y), __fmul_rn(k.y, r.x))));
        fv = __halves2half2(__float2half_rn(v.x), __float2half_rn(v.y));
        *reinterpret_cast<__half2 *>(kc + at) = fk;
        *reinterpret_cast<__half2 *>(vc + at) = fv;
    }
    float m[2], l[2], acc[2][DPL];                       // a warp's heads: warp and, with more than 16 heads to a KV head, warp + 16
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        m[h] = -CUDART_INF_F;
        l[h] = 0.f;
#pragma unroll
        for (int i = 0; i < DPL; ++i) acc[h][i] = 0.f;
    }
    bool ok = true;
    for (int k0 = key_lo; k0 < key_hi; k0 += STEP_KEYS) {
        if (!ready) {
            __syncthreads();                             // the chunk before has been read
            step_fetch_kv(smem_u32(kv), kc, vc, KV, HD, kvh, k0, key_hi, turn ? p : -1, kv_bar);
        }
        ready = false;
        if (fresh_here && p >= k0 && p < k0 + STEP_KEYS && ft < HD / 2) {
            *reinterpret_cast<__half2 *>(kv + (p - k0) * PITCH + 4 * ft) = fk;
            *reinterpret_cast<__half2 *>(kv + (STEP_KEYS + p - k0) * PITCH + 4 * ft) = fv;
        }
        ok = mbar_wait(kv_bar, phase) && ok;
        phase ^= 1u;
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int g = warp + SMALL_WARPS * h;
            if (g >= G) break;
            const float *q = qs + g * HD;
            const int key = k0 + lane;
            float s = -CUDART_INF_F;
            if (key < key_hi) {
                const uint4 *kr = reinterpret_cast<const uint4 *>(kv + lane * PITCH);
                float dot = 0.f;
#pragma unroll
                for (int c = 0; c < HD / 8; ++c) {
                    const uint4 u = kr[c];
                    const __half2 *hp = reinterpret_cast<const __half2 *>(&u);
                    const float4 q0 = *reinterpret_cast<const float4 *>(q + 8 * c), q1 = *reinterpret_cast<const float4 *>(q + 8 * c + 4);
                    const float qv[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 kf = __half22float2(hp[e]);
                        dot = fmaf(qv[2 * e], kf.x, dot);
                        dot = fmaf(qv[2 * e + 1], kf.y, dot);
                    }
                }
                s = dot * a.scale;
            }
            float cm = s;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
            const float m_new = fmaxf(m[h], cm);
            const float corr = expf(m[h] - m_new);       // 0 on the first chunk (m = -inf)
            const float pr = key < key_hi ? expf(s - m_new) : 0.f;
            float ps = pr;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, o);
            l[h] = l[h] * corr + ps;
#pragma unroll
            for (int i = 0; i < DPL; ++i) acc[h][i] *= corr;
            const int nk = min(32, key_hi - k0);
            const uint8_t *const vr = kv + STEP_KEYS * PITCH + 2 * DPL * lane;
#pragma unroll 8
            for (int j = 0; j < nk; ++j) {
                const float pj = __shfl_sync(0xffffffffu, pr, j);
                if (DPL == 4) {
                    const uint2 u = *reinterpret_cast<const uint2 *>(vr + j * PITCH);
                    const float2 x = __half22float2(*reinterpret_cast<const __half2 *>(&u.x));
                    const float2 y = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
                    acc[h][0] = fmaf(pj, x.x, acc[h][0]); acc[h][1] = fmaf(pj, x.y, acc[h][1]);
                    acc[h][DPL - 2] = fmaf(pj, y.x, acc[h][DPL - 2]); acc[h][DPL - 1] = fmaf(pj, y.y, acc[h][DPL - 1]);
                } else {
                    const float2 x = __half22float2(*reinterpret_cast<const __half2 *>(vr + j * PITCH));
                    acc[h][0] = fmaf(pj, x.x, acc[h][0]); acc[h][1] = fmaf(pj, x.y, acc[h][1]);
                }
            }
            m[h] = m_new;
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int g = warp + SMALL_WARPS * h;
        if (g >= G) break;
        float *pp = a.part + ((size_t)(kvh * G + g) * a.splits + z) * (HD + 2);
#pragma unroll
        for (int i = 0; i < DPL; ++i) pp[DPL * lane + i] = acc[h][i];
        if (lane == 0) { pp[HD] = m[h]; pp[HD + 1] = l[h]; }
    }
    return ok;
}
// the first ns shares of a KV head, combined and quantised to Q8_0 (attention_merge_q8_0_kernel)
template <int HD>
__device__ __forceinline__ void step_merge(const StepArgs &a, int kvh, int ns) {
    constexpr int DPL = HD / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, G = a.H / a.KV;
    for (int g = warp; g < G; g += SMALL_WARPS) {
        const int hh = kvh * G + g;
        const float *pp = a.part + (size_t)hh * a.splits * (HD + 2);
        // the first shares' sums are on their way before the largest score of all is known
        constexpr int AHEAD = 4;
        float lz[AHEAD], mz[AHEAD], v[AHEAD][DPL];
        auto fetch = [&](int z0) {
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) {
                const float *pz = pp + min(z0 + i, ns - 1) * (HD + 2);
                lz[i] = __ldcg(pz + HD + 1);
                mz[i] = __ldcg(pz + HD);
#pragma unroll
                for (int d = 0; d < DPL; ++d) v[i][d] = __ldcg(pz + DPL * lane + d);
            }
        };
        fetch(0);
        float mx = -CUDART_INF_F;
        for (int z = lane; z < ns; z += 32) mx = fmaxf(mx, __ldcg(pp + z * (HD + 2) + HD));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        float l = 0.f, acc[DPL];
#pragma unroll
        for (int i = 0; i < DPL; ++i) acc[i] = 0.f;
        for (int z0 = 0; z0 < ns; z0 += AHEAD) {
            if (z0 > 0) fetch(z0);
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) {
                if (z0 + i >= ns || lz[i] == 0.f) continue;
                const float wz = expf(mz[i] - mx);
                l = fmaf(wz, lz[i], l);
#pragma unroll
                for (int d = 0; d < DPL; ++d) acc[d] = fmaf(wz, v[i][d], acc[d]);
            }
        }
        const float inv = 1.0f / l;
        float amax = 0.f;
#pragma unroll
        for (int i = 0; i < DPL; ++i) {
            acc[i] *= inv;
            amax = fmaxf(amax, fabsf(acc[i]));
        }
#pragma unroll
        for (int o = 16 / DPL; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        const float dd = __fdiv_rn(amax, 127.f), id = dd != 0.f ? __fdiv_rn(1.0f, dd) : 0.f;
#pragma unroll
        for (int i = 0; i < DPL; ++i) a.aq[(size_t)hh * HD + DPL * lane + i] = (int8_t)roundf(__fmul_rn(acc[i], id));
        if (lane % (32 / DPL) == 0) a.ad[(hh * HD + DPL * lane) / 32] = __half2float(__float2half_rn(dd));
    }
}

template <int GU, int DN, SmallSums SUMS>
__global__ void __launch_bounds__(SMALL_THREADS, 1) decoder_step_kernel(const StepArgs a) {
    // a staging area per warp | quantised row [max(D, H HD)] and its scales | rotated heads [G][HD] | x [D] | packed input row | packed
    // SwiGLU rows | probabilities and scores.  From x on the memory holds a chunk of keys and values while attention runs.
    extern __shared__ __align__(128) uint8_t dyn[];
    __shared__ float s_part[SMALL_WARPS], s_w[SMALL_PAIRS];
    __shared__ int s_ids[SMALL_PAIRS], s_late;
    __shared__ __align__(8) uint64_t s_bars[SMALL_WARPS][SMALL_SLOTS];
    __shared__ unsigned s_last;
    __shared__ unsigned long long s_best[SMALL_WARPS];
    __shared__ float2 s_rot[64];
    __shared__ __align__(8) uint64_t s_kv_bar;
    __shared__ __align__(16) uint8_t s_layer_raw[sizeof(StepLayer)];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, D = a.D, QO = a.H * a.HD, G = a.H / a.KV;
    const int widest = D > QO ? D : QO, cols = (a.H + 2 * a.KV) * a.HD, rbd = D / 32 * 34, rbo = QO / 32 * 34;
    const StepLayer &s_layer = *reinterpret_cast<const StepLayer *>(s_layer_raw);
    const SmallArgs &moe = s_layer.moe;
    SmallShared s;
    s.stage = smem_u32(dyn) + (uint32_t)(warp * a.stage);
    int8_t *const xq = reinterpret_cast<int8_t *>(dyn + SMALL_WARPS * a.stage);
    float *const xd = reinterpret_cast<float *>(xq + widest);
    float *const qs = xd + ((widest / 32 + 3) & ~3);
    float *const x = qs + G * a.HD;
    uint8_t *const kv = reinterpret_cast<uint8_t *>(x);
    s.q8x = reinterpret_cast<uint8_t *>(x + D);
    s.q8f = s.q8x + q8row_stride(D);
    s.prob = nullptr;                                    // set per layer: it follows the SwiGLU rows
    s.ids = s_ids; s.w = s_w; s.part = s_part;
    auto load_layer = [&](int l) {                       // the CTA's copy of a layer's table entry
        __syncthreads();
        for (int i = tid; i < (int)(sizeof(StepLayer) / 4); i += SMALL_THREADS)
            reinterpret_cast<uint32_t *>(s_layer_raw)[i] = reinterpret_cast<const uint32_t *>(a.layers + l)[i];
        __syncthreads();
    };
    s.bars = s_bars[warp]; s.phase = 0; s.late = &s_late;
    if (tid == 0) mbar_init(&s_kv_bar, 1);
    small_init(s_bars, &s_late);
    load_layer(0);
    step_prefetch(s, s_layer.wqkv, cols, rbd, a.depth_q);
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    const int p = *a.pos;
    // the angles as the reference builds them: pos * scale * scale * ..., in f32
    if (tid < a.HD / 2) {
        float ang = (float)p;
        for (int i = 0; i < tid; ++i) ang = __fmul_rn(ang, a.theta_scale);
        s_rot[tid] = make_float2(cosf(ang), sinf(ang));
    }
    int tok = *a.token;
    tok = tok < 0 ? 0 : tok >= a.vocab ? a.vocab - 1 : tok;
    for (int i = tid; i < D; i += SMALL_THREADS) {
        const uint8_t *blk = a.embd + (size_t)tok * rbd + (size_t)(i >> 5) * 34;
        const float v = __half2float(__ushort_as_half((unsigned short)(blk[0] | (blk[1] << 8)))) * (float)(int8_t)blk[2 + (i & 31)];
        x[i] = v;
        if (blockIdx.x == 0) a.h[i] = v;                 // read by other CTAs after the first barrier at the earliest
    }
    __syncthreads();
    unsigned n_bar = 0;
    // a wait that runs out is seen through every layer's context, as it would be after the separate launches of that layer
    auto expired = [&]() {
        for (int l = 0; l < a.n_layers; ++l) atomicExch(a.layers[l].moe.err, 21);
    };
    auto barrier = [&]() { small_grid_barrier(a.bar, ++n_bar, expired); };
    auto load_h = [&]() {
        for (int i = tid; i < D / 4; i += SMALL_THREADS) reinterpret_cast<float4 *>(x)[i] = __ldcg(reinterpret_cast<const float4 *>(a.h) + i);
        __syncthreads();
    };
    uint32_t kv_phase = 0;
    int n_keys, per, ns;
    step_shares(a, p, n_keys, per, ns);
    for (int l = 0; l < a.n_layers; ++l) {
        const size_t layer_kv = (size_t)l * a.max_ctx * a.KV * a.HD;
        if (l > 0) load_h();
        s.prob = reinterpret_cast<float *>(s.q8f + moe.K * q8row_stride(moe.F));
        step_norm(x, s_layer.attn_norm, D, a.eps, s_part);
        step_quantise(x, xq, xd, D);
        if (blockIdx.x < a.KV * ns) {       // x is free: the first keys and values that this CTA will meet
            const int z = blockIdx.x % ns;
            step_fetch_kv(smem_u32(kv), a.kc + layer_kv, a.vc + layer_kv, a.KV, a.HD, blockIdx.x / ns, min(n_keys, z * per * 32),
                          min(n_keys, (z + 1) * per * 32), p < a.max_ctx ? p : -1, &s_kv_bar);
        }
        step_rows(s, s_layer.wqkv, cols, rbd, a.depth_q, xq, xd, [&](int o, float v) { a.qkv[o] = v; });
        step_prefetch(s, s_layer.wo, D, rbo, a.depth_o);
        small_prefetch_router(moe);
        barrier();
        // ---- attention: a CTA per share of a KV head that has keys ----
        {
            for (int u = blockIdx.x; u < a.KV * ns; u += gridDim.x) {
                const int kvh = u / ns, z = u % ns;
                const bool first = u == (int)blockIdx.x;
                if (!first) __syncthreads();             // qs is still read
                const bool ok = a.HD == 128 ? step_attention<128>(a, a.kc + layer_kv, a.vc + layer_kv, kvh, z, p, qs, s_rot, kv, &s_kv_bar, kv_phase, first)
                                            : step_attention<64>(a, a.kc + layer_kv, a.vc + layer_kv, kvh, z, p, qs, s_rot, kv, &s_kv_bar, kv_phase, first);
                if (!ok) s_late = 1;
                __syncthreads();
                // one thread's release and acquire order what the CTA wrote and what it reads next
                if (tid == 0) asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(s_last) : "l"(a.head_ticket + kvh) : "memory");
                __syncthreads();
                if (s_last == (unsigned)ns - 1) {
                    if (a.HD == 128) step_merge<128>(a, kvh, ns); else step_merge<64>(a, kvh, ns);
                    if (tid == 0) a.head_ticket[kvh] = 0u;
                }
            }
        }
        barrier();
        // ---- output projection, added to the residual stream ----
        for (int i = tid; i < QO / 16; i += SMALL_THREADS) reinterpret_cast<uint4 *>(xq)[i] = __ldcg(reinterpret_cast<const uint4 *>(a.aq) + i);
        for (int i = tid; i < QO / 32; i += SMALL_THREADS) xd[i] = __ldcg(a.ad + i);
        __syncthreads();
        step_rows(s, s_layer.wo, D, rbo, a.depth_o, xq, xd, [&](int o, float v) { a.h[o] = __ldcg(a.h + o) + v; });
        barrier();
        // ---- MoE block ----
        load_h();
        step_norm(x, s_layer.ffn_norm, D, a.eps, s_part);
        small_logits<GU>(moe, s, x);
        barrier();
        small_gate_up<GU, SUMS>(moe, s);
        small_prefetch_down<SUMS != SUMS_BLOCKS>(moe, s);
        barrier();
        small_down<DN, SUMS>(moe, s);
        if (s_layer.leave_state && blockIdx.x == gridDim.x - 1) {
            __syncthreads();
            for (int i = tid; i < D; i += SMALL_THREADS) a.xn[i] = x[i];
            small_leave_state(moe, s);
        }
        if (l + 1 < a.n_layers) {
            load_layer(l + 1);
            step_prefetch(s, s_layer.wqkv, cols, rbd, a.depth_q);
        } else {
            step_prefetch(s, a.head, a.vocab, rbd, a.depth_q);
        }
        barrier();
    }
    // ---- output head, arg-max (lowest index on ties) ----
    load_h();
    step_norm(x, a.out_norm, D, a.eps, s_part);
    step_quantise(x, xq, xd, D);
    unsigned long long best = 0ull;
    step_rows(s, a.head, a.vocab, rbd, a.depth_q, xq, xd, [&](int o, float v) {
        a.logits[o] = v;
        if (!isnan(v)) {
            const unsigned u = __float_as_uint(__fadd_rn(v, 0.f));
            const unsigned long long key = ((unsigned long long)((u >> 31) ? ~u : u | 0x80000000u) << 32) | (0xffffffffu - (unsigned)o);
            best = key > best ? key : best;
        }
    });
    if (lane == 0) s_best[warp] = best;
    __syncthreads();
    if (tid == 0) {
        if (s_late) expired();
        for (int i = 1; i < SMALL_WARPS; ++i) best = s_best[i] > best ? s_best[i] : best;
        if (best) atomicMax(a.best, best);
        __threadfence();
        // the last CTA to leave ends the step
        if (atomicAdd(a.bar + 1, 1u) == gridDim.x - 1) {
            __threadfence();
            const unsigned long long key = *reinterpret_cast<volatile unsigned long long *>(a.best);
            *a.next = key ? (int32_t)(0xffffffffu - (unsigned)key) : 0;
            *a.pos = p + 1;
            *a.best = 0ull;
            a.bar[0] = 0u;
            a.bar[1] = 0u;
        }
    }
}

}  // namespace zmoe
