// decoder.cu -- the dense kernels around the MoE block and a decoder step built from them: RMSNorm, dense
// Q8_0 matmul (attention projections, output head), RoPE, grouped-query attention over an f16 KV cache,
// greedy sampling.  With these the fifth benchmark configuration (a full random-init MoE decoder) runs end to
// end on the device.
//
// What each piece follows in the reference:
//   RMSNorm     y = x * rsqrt(mean(x^2) + eps) * w            kernels/math/rmsnorm.cu:6-78 (launch_rmsnorm)
//   Q8_0        34-byte blocks {fp16 d; int8 q[32]}, w = d*q  kernels/quant/q8_0_matmul.cu:20-60,189-221
//   RoPE        interleaved pairs (2j, 2j+1), angle pos * theta^(-2j/dim) built by repeated multiplication
//                                                             models/base/rope.hpp:52-118 (no YaRN: ext_factor 0)
//   attention   scores q.k / sqrt(head_dim), max-subtracted softmax, sum p*v; q head h reads kv head
//               h / (n_heads / n_kv_heads)                     core/attention_layer.cpp:2633-2690
// As everywhere in this library the matmul follows the reference's CPU arithmetic (ggml MUL_MAT): the
// activation row is quantised too (Q8_0 per 32 values) and blocks are multiplied in integers; the
// reference's own CUDA kernel multiplies f32 activations by dequantised weights.
#include <cuda_fp16.h>
#include <math_constants.h>

#include <cmath>
#include <mutex>
#include <new>
#include <type_traits>
#include <vector>

#include "quant_units.cuh"
#include "zmoe_internal.h"

using namespace zmoe;

namespace {

inline int cu(cudaError_t e) { return e == cudaSuccess ? ZMOE_OK : ZMOE_ERR_CUDA; }

// ---------------------------------------------------------------------------
// RMSNorm: one CTA per row
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) rmsnorm_kernel(float *__restrict__ y, const float *__restrict__ x,
                                                      const float *__restrict__ w, int D, float eps) {
    __shared__ float s_part[8];
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float4 *xv = reinterpret_cast<const float4 *>(x + (size_t)row * D);
    const float4 *wv = reinterpret_cast<const float4 *>(w);
    float4 *yv = reinterpret_cast<float4 *>(y + (size_t)row * D);
    float ss = 0.f;
    for (int i = tid; i < D / 4; i += 256) {
        const float4 v = xv[i];
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) s_part[warp] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) tot += s_part[i];
    const float inv = rsqrtf(tot / (float)D + eps);
    for (int i = tid; i < D / 4; i += 256) {
        const float4 v = xv[i], g = wv[i];
        yv[i] = make_float4(v.x * inv * g.x, v.y * inv * g.y, v.z * inv * g.z, v.w * inv * g.w);
    }
}

// RMSNorm followed by the Q8_0 quantiser in one launch (the normed row only feeds a Q8_0 matmul): one CTA per
// row, a thread owns four consecutive elements, the eight threads of a 32-element block share its maximum.
// Same arithmetic, in the same order, as rmsnorm_kernel followed by quantize_q8_0_kernel.
__global__ void __launch_bounds__(256) rmsnorm_q8_0_kernel(int8_t *__restrict__ q, float *__restrict__ d,
                                                           const float *__restrict__ x, const float *__restrict__ w, int D,
                                                           float eps) {
    __shared__ float s_part[8];
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float4 *xv = reinterpret_cast<const float4 *>(x + (size_t)row * D);
    const float4 *wv = reinterpret_cast<const float4 *>(w);
    float ss = 0.f;
    for (int i = tid; i < D / 4; i += 256) {
        const float4 v = xv[i];
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) s_part[warp] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) tot += s_part[i];
    const float inv = rsqrtf(tot / (float)D + eps);
    const int nb = D / 32;
    // D is a multiple of 32: whole groups of eight threads run each iteration together
    for (int i = tid; i < D / 4; i += 256) {
        const float4 v = xv[i], g = wv[i];
        const float y0 = v.x * inv * g.x, y1 = v.y * inv * g.y, y2 = v.z * inv * g.z, y3 = v.w * inv * g.w;
        float amax = fmaxf(fmaxf(fabsf(y0), fabsf(y1)), fmaxf(fabsf(y2), fabsf(y3)));
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        const float dd = __fdiv_rn(amax, 127.f);
        const float id = dd != 0.f ? __fdiv_rn(1.0f, dd) : 0.f;
        char4 o4;
        o4.x = (signed char)roundf(__fmul_rn(y0, id)); o4.y = (signed char)roundf(__fmul_rn(y1, id));
        o4.z = (signed char)roundf(__fmul_rn(y2, id)); o4.w = (signed char)roundf(__fmul_rn(y3, id));
        reinterpret_cast<char4 *>(q + (size_t)row * D)[i] = o4;
        if ((tid & 7) == 0) d[(size_t)row * nb + (i >> 3)] = __half2float(__float2half_rn(dd));
    }
}

// ---------------------------------------------------------------------------
// Q8_0 activation quantiser: one warp per block of 32 values.  q int8 [rows, I], d f32 [rows, I / 32] holds
// the fp16-rounded scale (what the dot multiplies with).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) quantize_q8_0_kernel(const float *__restrict__ x, int ldx, int8_t *__restrict__ q,
                                                            float *__restrict__ d, int rows, int I) {
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    const int nb = I / 32, lane = threadIdx.x & 31;
    for (long blk = (long)blockIdx.x * 8 + (threadIdx.x >> 5); blk < (long)rows * nb; blk += (long)gridDim.x * 8) {
        const int r = (int)(blk / nb), b = (int)(blk % nb);
        const float v = x[(size_t)r * ldx + 32 * b + lane];
        float amax = fabsf(v);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        const float dd = __fdiv_rn(amax, 127.f);
        const float id = dd != 0.f ? __fdiv_rn(1.0f, dd) : 0.f;
        q[(size_t)r * I + 32 * b + lane] = (int8_t)roundf(__fmul_rn(v, id));
        if (lane == 0) d[(size_t)r * nb + b] = __half2float(__float2half_rn(dd));
    }
}

// ---------------------------------------------------------------------------
// Dense Q8_0 matmul: y[s, o] (+)= sum over blocks of (q_w . q_x) * d_w * d_x.  A warp owns an output row: it
// stages the row's bytes in shared memory with coalesced 16-byte loads, lanes take blocks, the activation
// chunk (up to SC rows) sits in shared memory for the whole CTA, so a weight row is read once per SC rows.  A warp's first
// weight row is staged before the wait for the kernel that writes the activations: every launch here follows one of this
// library's kernels that itself waited for its predecessor, so whatever wrote the weights has ended.  With the one-row
// instantiation, the quantising merge and the position moved by the arg-max, a decode step of two layers and a head of
// 8192 took 190 -> 158 us as separate launches (one kernel where decoder_step.cuh takes it: 139).
// ---------------------------------------------------------------------------
constexpr int MM_WARPS = 8;
template <int SC>
__global__ void __launch_bounds__(32 * MM_WARPS) q8_0_matmul_kernel(float *__restrict__ y, int ldy,
                                                                    const uint8_t *__restrict__ w, size_t w_bytes,
                                                                    const int8_t *__restrict__ xq,
                                                                    const float *__restrict__ xd, int S, int I, int O,
                                                                    int accumulate) {
    extern __shared__ __align__(16) uint8_t sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = I / 32, rb = nb * 34;
    const int rbs = (rb + 32 + 15) & ~15;                   // row buffer: room for the offset from a 16-byte boundary
    int8_t *aq = reinterpret_cast<int8_t *>(sm);            // [SC][I]
    float *ad = reinterpret_cast<float *>(sm + (size_t)SC * I);   // [SC][nb]
    uint8_t *wrow = sm + (size_t)SC * I + (((size_t)SC * nb * 4 + 15) & ~(size_t)15) + (size_t)warp * rbs;
    const uint32_t wrow_s = smem_u32(wrow);
    const size_t w_end16 = w_bytes & ~(size_t)15;           // 16-byte loads stay below this offset
    auto stage_row = [&](int o) {
        const size_t g = (size_t)o * rb;
        const int off = (int)(g & 15);
        const size_t g0 = g - off;
        const int nchunk = (off + rb + 15) / 16;
        for (int c = lane; c < nchunk; c += 32) {
            const size_t at = g0 + 16 * (size_t)c;
            uint4 v;
            if (at + 16 <= w_end16) {
                v = *reinterpret_cast<const uint4 *>(w + at);
            } else {   // the last bytes of the tensor
                __align__(16) uint8_t tmp[16];
                for (int i = 0; i < 16; ++i) tmp[i] = at + i < w_bytes ? w[at + i] : 0;
                v = *reinterpret_cast<uint4 *>(tmp);
            }
            reinterpret_cast<uint4 *>(wrow)[c] = v;
        }
    };
    const int o_first = blockIdx.x * MM_WARPS + warp;
    if (o_first < O) stage_row(o_first);
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    for (int s0 = 0; s0 < S; s0 += SC) {
        const int ns = min(SC, S - s0);
        __syncthreads();
        for (int i = tid; i < ns * I / 16; i += blockDim.x)
            reinterpret_cast<uint4 *>(aq)[i] = reinterpret_cast<const uint4 *>(xq + (size_t)s0 * I)[i];
        for (int i = tid; i < ns * nb; i += blockDim.x) ad[i] = xd[(size_t)s0 * nb + i];
        __syncthreads();
        for (int o = o_first; o < O; o += gridDim.x * MM_WARPS) {
            const int off = (int)(((size_t)o * rb) & 15);
            if (s0 > 0 || o != o_first) stage_row(o);
            __syncwarp();
            float acc[SC];
#pragma unroll
            for (int s = 0; s < SC; ++s) acc[s] = 0.f;
            for (int b = lane; b < nb; b += 32) {
                const uint32_t blk = wrow_s + off + 34 * b;
                const float dw = half_bits_to_float(lds16(blk));
                uint32_t qw[8];
                lds32xN_any<2, 8>(blk + 2, qw);
#pragma unroll
                for (int s = 0; s < SC; ++s) {
                    if (s < ns) {
                        const uint4 a0 = *reinterpret_cast<const uint4 *>(aq + (size_t)s * I + 32 * b);
                        const uint4 a1 = *reinterpret_cast<const uint4 *>(aq + (size_t)s * I + 32 * b + 16);
                        int sum = __dp4a((int)qw[0], (int)a0.x, 0);
                        sum = __dp4a((int)qw[1], (int)a0.y, sum);
                        sum = __dp4a((int)qw[2], (int)a0.z, sum);
                        sum = __dp4a((int)qw[3], (int)a0.w, sum);
                        sum = __dp4a((int)qw[4], (int)a1.x, sum);
                        sum = __dp4a((int)qw[5], (int)a1.y, sum);
                        sum = __dp4a((int)qw[6], (int)a1.z, sum);
                        sum = __dp4a((int)qw[7], (int)a1.w, sum);
                        acc[s] = __fadd_rn(acc[s], __fmul_rn((float)sum, __fmul_rn(dw, ad[s * nb + b])));
                    }
                }
            }
#pragma unroll
            for (int s = 0; s < SC; ++s) {
#pragma unroll
                for (int o2 = 16; o2 > 0; o2 >>= 1) acc[s] += __shfl_xor_sync(0xffffffffu, acc[s], o2);
            }
            if (lane == 0) {
#pragma unroll
                for (int s = 0; s < SC; ++s)
                    if (s < ns) {
                        float *dst = y + (size_t)(s0 + s) * ldy + o;
                        *dst = accumulate ? *dst + acc[s] : acc[s];
                    }
            }
            __syncwarp();
        }
    }
}

// ---------------------------------------------------------------------------
// The same for more than eight rows: BM weight rows x BN activation rows per CTA on the int8 tensor cores
// (mma.sync m16n8k32: one Q8_0 block per instruction, so a block's exact integer sum comes out before its two scales
// are applied).  The kernel above multiplies eight rows per pass over the weights with dp4a, 32 of them per eight
// outputs of a warp's lanes; at 512 rows it took 763 us for a [5120 x 2048] projection (64 passes), this one 56, bound by
// the instructions per output and block that apply the scales.  Eight blocks (272 bytes of a weight row, 256 of an
// activation row) per stage, three stages of asynchronous copies; the pitch of 272 bytes puts a fragment's eight rows into
// different banks.  A weight block starts on a word only if its number is odd (2 + 34 b bytes): even ones are read as two
// words and shifted.  The integer accumulators start at the bit pattern of 1.5 * 2^23, which makes them read as the float
// 1.5 * 2^23 + sum: one exact subtraction converts them.
// ---------------------------------------------------------------------------
constexpr int MQ_KB = 8, MQ_NST = 3, MQ_PITCH = 34 * MQ_KB, MQ_DPITCH = 12;   // floats between the scales of activation rows

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// 16 bytes, or 16 zeros without reading anything
__device__ __forceinline__ void cp_async16_or_zeros(uint32_t dst, const void *src, bool read) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(read ? 16 : 0) : "memory");
}
__device__ __forceinline__ void mma_s8(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int BM, int BN>
__host__ __device__ constexpr int mq_stage_bytes() { return (BM + BN) * MQ_PITCH + BN * MQ_DPITCH * 4; }

// RAGGED: activation rows that are not there arrive as zeros.  With copies of the last row in their place every CTA read one
// row up to 55 times over: 9, 65 and 600 rows against a [37984 x 1024] head took 143, 169 and 310 us (64 rows: 35), and 33, 57
// and 248 with the zeros.  The test costs full tiles 1 % (5 % at 700 rows of [2048 x 7168]): they, and tiles that lack an
// eighth of their rows at most, keep the plain copies.
template <int BM, int BN, bool RAGGED>
__global__ void __launch_bounds__(128) q8_0_mma_kernel(float *__restrict__ y, int ldy, const uint8_t *__restrict__ w,
                                                       const int8_t *__restrict__ xq, const float *__restrict__ xd, int S,
                                                       int I, int O, int accumulate) {
    extern __shared__ __align__(16) uint8_t sm[];
    constexpr int STAGE = mq_stage_bytes<BM, BN>(), MT = BM / 32, NT = BN / 16;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c = lane & 3;
    const int nb = I / 32, nst = nb / MQ_KB;
    const size_t rb = (size_t)nb * 34;
    const int o0 = blockIdx.x * BM, s0 = blockIdx.y * BN;
    const int wm = (warp >> 1) * (BM / 2), wn = (warp & 1) * (BN / 2);
    const uint32_t base = smem_u32(sm);
    auto load_w = [&](int st) {
        const uint32_t dst = base + (st % MQ_NST) * STAGE;
        for (int i = tid; i < BM * 17; i += 128) {
            const int r = i / 17, k = i % 17;
            cp_async16(dst + r * MQ_PITCH + 16 * k, w + (size_t)min(o0 + r, O - 1) * rb + (size_t)st * MQ_PITCH + 16 * k);
        }
    };
    auto copy_x = [&](uint32_t dst, const void *src, int r) {
        if (RAGGED) cp_async16_or_zeros(dst, src, s0 + r < S);
        else cp_async16(dst, src);
    };
    auto load_x = [&](int st) {
        const uint32_t dst = base + (st % MQ_NST) * STAGE + BM * MQ_PITCH;
        for (int i = tid; i < BN * 16; i += 128) {
            const int r = i >> 4, k = i & 15;
            copy_x(dst + r * MQ_PITCH + 16 * k, xq + (size_t)min(s0 + r, S - 1) * I + st * (32 * MQ_KB) + 16 * k, r);
        }
        for (int i = tid; i < BN * 2; i += 128) {
            const int r = i >> 1, k = i & 1;
            copy_x(dst + BN * MQ_PITCH + r * MQ_DPITCH * 4 + 16 * k, xd + (size_t)min(s0 + r, S - 1) * nb + st * MQ_KB + 4 * k, r);
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    for (int st = 0; st < MQ_NST - 1; ++st) {
        if (st < nst) { load_w(st); load_x(st); }
        commit();
    }
    float acc[MT][NT][4], comp[MT][NT][4];     // sums of the stages, with Kahan's compensation
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[i][j][k] = comp[i][j][k] = 0.f;
    for (int st = 0; st < nst; ++st) {
        asm volatile("cp.async.wait_group %0;" ::"n"(MQ_NST - 2) : "memory");
        __syncthreads();                       // stage st has landed for all, and the slot refilled next is free
        if (st + MQ_NST - 1 < nst) { load_w(st + MQ_NST - 1); load_x(st + MQ_NST - 1); }
        commit();
        const uint32_t ws = base + (st % MQ_NST) * STAGE + (wm + g) * MQ_PITCH;
        const uint32_t xs = base + (st % MQ_NST) * STAGE + (BM + wn + g) * MQ_PITCH + 4 * c;
        const uint32_t ds = base + (st % MQ_NST) * STAGE + (BM + BN) * MQ_PITCH + (wn + 2 * c) * MQ_DPITCH * 4;
        // Sums of eight blocks first, then the compensated sum of those: the kernel above adds lanes pairwise, and a chain of
        // all blocks would round more than that (measured against 64 bits: 7.8e-8 without the compensation, 7.1e-8 there)
        float part[MT][NT][4];
#pragma unroll
        for (int b = 0; b < MQ_KB; ++b) {
            uint32_t a[MT][4];
            float dw[MT][2];
#pragma unroll
            for (int i = 0; i < MT; ++i) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t row = ws + (16 * i + 8 * h) * MQ_PITCH + 34 * b;
                    dw[i][h] = half_bits_to_float(lds16(row));
                    if (b & 1) {
                        a[i][h] = lds32(row + 2 + 4 * c);
                        a[i][2 + h] = lds32(row + 18 + 4 * c);
                    } else {
                        a[i][h] = __funnelshift_r(lds32(row + 4 * c), lds32(row + 4 + 4 * c), 16);
                        a[i][2 + h] = __funnelshift_r(lds32(row + 16 + 4 * c), lds32(row + 20 + 4 * c), 16);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const uint32_t b0 = lds32(xs + 8 * j * MQ_PITCH + 32 * b), b1 = lds32(xs + 8 * j * MQ_PITCH + 32 * b + 16);
                const float dx0 = __uint_as_float(lds32(ds + 8 * j * MQ_DPITCH * 4 + 4 * b));
                const float dx1 = __uint_as_float(lds32(ds + (8 * j + 1) * MQ_DPITCH * 4 + 4 * b));
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    int t[4] = {0x4B400000, 0x4B400000, 0x4B400000, 0x4B400000};
                    mma_s8(t, a[i], b0, b1);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float sum = __int_as_float(t[k]) - 12582912.f;
                        const float d = __fmul_rn(dw[i][k >> 1], (k & 1) ? dx1 : dx0);
                        part[i][j][k] = b == 0 ? __fmul_rn(sum, d) : fmaf(sum, d, part[i][j][k]);
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float v = __fsub_rn(part[i][j][k], comp[i][j][k]), t = __fadd_rn(acc[i][j][k], v);
                    // An infinite scale makes the sum infinite and its compensation NaN; the sum has to stay what it is.  The
                    // maximum drops a NaN, and finite scales never come near its bound: a block is at most 32 * 127 * 127 *
                    // 65504^2 = 2^51, so is the compensation of fewer than 2^24 of them.
                    comp[i][j][k] = fmaxf(__fsub_rn(__fsub_rn(t, acc[i][j][k]), v), -0x1p105f);
                    acc[i][j][k] = t;
                }
    }
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int o = o0 + wm + 16 * i + g + 8 * (k >> 1), r = s0 + wn + 8 * j + 2 * c + (k & 1);
                if (o < O && r < S) {
                    float *dst = y + (size_t)r * ldy + o;
                    *dst = accumulate ? *dst + acc[i][j][k] : acc[i][j][k];
                }
            }
}

// dequantised rows of a Q8_0 table for a list of row numbers (token embedding): one CTA per token
__global__ void __launch_bounds__(256) embed_q8_0_kernel(const int32_t *__restrict__ tokens, const uint8_t *__restrict__ w,
                                                         float *__restrict__ h, int D, int vocab) {
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    const int t = blockIdx.x;
    int tok = tokens[t];
    tok = tok < 0 ? 0 : tok >= vocab ? vocab - 1 : tok;
    const uint8_t *row = w + (size_t)tok * (D / 32) * 34;
    for (int i = threadIdx.x; i < D; i += blockDim.x) {
        const uint8_t *blk = row + (i >> 5) * 34;
        const float d = __half2float(__ushort_as_half((unsigned short)(blk[0] | (blk[1] << 8))));
        h[(size_t)t * D + i] = d * (float)(int8_t)blk[2 + (i & 31)];
    }
}

// ---------------------------------------------------------------------------
// RoPE on q and k (in place, interleaved pairs) and append of k, v to the f16 cache.  qkv: [T, (H + 2 KV) * hd]
// rows of q | k | v.  Token t sits at position *pos + t.  grid (T, ceil((H + KV) / HEADS)), hd / 2 threads: a thread turns its pair of HEADS heads,
// whose values are on their way while it builds the angle.  What bounds it: the angle, up to 63 products in a row and a sine and a cosine; a head at a
// time, every head built it anew (512 tokens of 32 + 4 heads: 21.0 us, 5.8 now).
// late: the attention behind it may not be placed before this kernel's work is done (rope_holds_attention).
// ---------------------------------------------------------------------------
constexpr int ROPE_TOKENS = 16;      // from so many tokens on the grid is large enough with six heads per CTA
template <int HEADS>
__global__ void rope_kv_kernel(float *__restrict__ qkv, __half *__restrict__ kc, __half *__restrict__ vc,
                               const int *__restrict__ pos, int H, int KV, int hd, float theta_scale, int max_ctx, int late) {
    pdl_wait_prior_grid();
    if (!late) pdl_launch_dependents();
    const int t = blockIdx.x, h0 = blockIdx.y * HEADS, j = threadIdx.x;
    const int p = *pos + t;
    if (p >= max_ctx) return;
    float *const row = qkv + (size_t)t * (H + 2 * KV) * hd;   // q heads, then k heads
    float2 x[HEADS], vv[HEADS];
#pragma unroll
    for (int i = 0; i < HEADS; ++i) {
        const int head = h0 + i;
        x[i] = vv[i] = make_float2(0.f, 0.f);
        if (head < H + KV) x[i] = *reinterpret_cast<const float2 *>(row + (size_t)head * hd + 2 * j);
        if (head >= H && head < H + KV) vv[i] = *reinterpret_cast<const float2 *>(row + (size_t)(head + KV) * hd + 2 * j);
    }
    // the angle as the reference builds it: pos * scale * scale * ... (j factors), all in f32, with
    // scale = theta_base^(-2 / head_dim) computed once on the host (as the reference's host code does)
    float ang = (float)p;
    for (int i = 0; i < j; ++i) ang = __fmul_rn(ang, theta_scale);
    const float c = cosf(ang), s = sinf(ang);
#pragma unroll
    for (int i = 0; i < HEADS; ++i) {
        const int head = h0 + i;
        if (head >= H + KV) break;
        const float ra = __fsub_rn(__fmul_rn(x[i].x, c), __fmul_rn(x[i].y, s)), rb = __fadd_rn(__fmul_rn(x[i].x, s), __fmul_rn(x[i].y, c));
        *reinterpret_cast<float2 *>(row + (size_t)head * hd + 2 * j) = make_float2(ra, rb);
        if (head >= H) {
            const size_t at = ((size_t)p * KV + (head - H)) * hd + 2 * j;
            *reinterpret_cast<__half2 *>(kc + at) = __halves2half2(__float2half_rn(ra), __float2half_rn(rb));
            *reinterpret_cast<__half2 *>(vc + at) = __halves2half2(__float2half_rn(vv[i].x), __float2half_rn(vv[i].y));
        }
    }
    if (late) pdl_launch_dependents();
}

// ---------------------------------------------------------------------------
// Grouped-query attention over the f16 cache, causal, keys split over CTAs.  grid (T, KV, NS); one warp per
// query head of the group.  Split z of a token takes the z-th share of its keys and leaves a partial
// (running maximum, sum of weights, weighted sum of V) in scratch; attention_merge_q8_0_kernel combines the shares.
// A lane owns one key of a 32-key chunk for the scores (the whole head_dim dot product, K row read as 16-byte
// pieces) and DPL output dimensions for the weighted sum of V; the softmax is the running-maximum form.
// ---------------------------------------------------------------------------
constexpr int ATTN_SPLITS = 16;
template <int HD>
__global__ void __launch_bounds__(1024) attention_kernel(const float *__restrict__ qkv, const __half *__restrict__ kc,
                                                         const __half *__restrict__ vc, float *__restrict__ part,
                                                         const int *__restrict__ pos, int H, int KV, float scale,
                                                         int max_ctx) {
    constexpr int DPL = HD / 32;
    extern __shared__ float q_s[];          // [warps][HD]
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    const int t = blockIdx.x, kvh = blockIdx.y, z = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = H / KV, h = kvh * G + warp;
    const int n_keys = min(*pos + t + 1, max_ctx);
    // this split's keys: whole chunks of 32, shared out evenly
    const int chunks = (n_keys + 31) / 32, per = (chunks + ATTN_SPLITS - 1) / ATTN_SPLITS;
    const int key_lo = min(n_keys, z * per * 32), key_hi = min(n_keys, (z + 1) * per * 32);
    const int ld = (H + 2 * KV) * HD;
    float *qs = q_s + warp * HD;
    for (int i = lane; i < HD; i += 32) qs[i] = qkv[(size_t)t * ld + (size_t)h * HD + i];
    __syncwarp();
    float m = -CUDART_INF_F, l = 0.f, acc[DPL];
#pragma unroll
    for (int i = 0; i < DPL; ++i) acc[i] = 0.f;
    for (int k0 = key_lo; k0 < key_hi; k0 += 32) {
        const int key = k0 + lane;
        float s = -CUDART_INF_F;
        if (key < key_hi) {
            const uint4 *kr = reinterpret_cast<const uint4 *>(kc + ((size_t)key * KV + kvh) * HD);
            float dot = 0.f;
#pragma unroll
            for (int c = 0; c < HD / 8; ++c) {
                const uint4 u = kr[c];
                const __half2 *hp = reinterpret_cast<const __half2 *>(&u);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 kf = __half22float2(hp[e]);
                    dot = fmaf(qs[8 * c + 2 * e], kf.x, dot);
                    dot = fmaf(qs[8 * c + 2 * e + 1], kf.y, dot);
                }
            }
            s = dot * scale;
        }
        float cm = s;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
        const float m_new = fmaxf(m, cm);
        const float corr = expf(m - m_new);          // 0 on the first chunk (m = -inf)
        const float pr = key < key_hi ? expf(s - m_new) : 0.f;
        float ps = pr;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, o);
        l = l * corr + ps;
#pragma unroll
        for (int i = 0; i < DPL; ++i) acc[i] *= corr;
        const int nk = min(32, key_hi - k0);
        for (int j = 0; j < nk; ++j) {
            const float pj = __shfl_sync(0xffffffffu, pr, j);
            const __half *vr = vc + ((size_t)(k0 + j) * KV + kvh) * HD + DPL * lane;
            if (DPL == 4) {
                const uint2 u = *reinterpret_cast<const uint2 *>(vr);
                const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u.x));
                const float2 b = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
                acc[0] = fmaf(pj, a.x, acc[0]); acc[1] = fmaf(pj, a.y, acc[1]);
                acc[2] = fmaf(pj, b.x, acc[2]); acc[3] = fmaf(pj, b.y, acc[3]);
            } else {
#pragma unroll
                for (int i = 0; i < DPL; ++i) acc[i] = fmaf(pj, __half2float(vr[i]), acc[i]);
            }
        }
        m = m_new;
    }
    // partial of (t, h, z): [HD values | m | l]
    float *pp = part + (((size_t)t * H + h) * ATTN_SPLITS + z) * (HD + 2);
#pragma unroll
    for (int i = 0; i < DPL; ++i) pp[DPL * lane + i] = acc[i];
    if (lane == 0) { pp[HD] = m; pp[HD + 1] = l; }
}

// out[t, h, :] = sum_z w_z * acc_z / sum_z w_z * l_z with w_z = exp(m_z - max m); one warp per (t, h); shares are
// added in ascending z (empty shares have l = 0 and m = -inf).  The row only feeds the Q8_0 output projection, so it is
// quantised here (the arithmetic of quantize_q8_0_kernel; the 32 / DPL lanes that hold a block share its maximum): a
// step of a few tokens is bound by its chain of launches, about 6 us each, and this takes one out per layer.
template <int HD>
__global__ void __launch_bounds__(256) attention_merge_q8_0_kernel(const float *__restrict__ part, int8_t *__restrict__ q,
                                                                   float *__restrict__ d, int TH) {
    constexpr int DPL = HD / 32;
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    const int th = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (th >= TH) return;
    const float *pp = part + (size_t)th * ATTN_SPLITS * (HD + 2);
    float mx = -CUDART_INF_F;
    for (int z = 0; z < ATTN_SPLITS; ++z) mx = fmaxf(mx, pp[z * (HD + 2) + HD]);
    float l = 0.f, acc[DPL];
#pragma unroll
    for (int i = 0; i < DPL; ++i) acc[i] = 0.f;
    for (int z = 0; z < ATTN_SPLITS; ++z) {
        const float lz = pp[z * (HD + 2) + HD + 1];
        if (lz == 0.f) continue;
        const float wz = expf(pp[z * (HD + 2) + HD] - mx);
        l = fmaf(wz, lz, l);
#pragma unroll
        for (int i = 0; i < DPL; ++i) acc[i] = fmaf(wz, pp[z * (HD + 2) + DPL * lane + i], acc[i]);
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
    const float dd = __fdiv_rn(amax, 127.f);
    const float id = dd != 0.f ? __fdiv_rn(1.0f, dd) : 0.f;
#pragma unroll
    for (int i = 0; i < DPL; ++i) q[(size_t)th * HD + DPL * lane + i] = (int8_t)roundf(__fmul_rn(acc[i], id));
    if (lane % (32 / DPL) == 0) d[((size_t)th * HD + DPL * lane) / 32] = __half2float(__float2half_rn(dd));
}

// ---------------------------------------------------------------------------
// The same for many tokens at once (a prompt): a CTA takes 64 query rows of one KV head (64 / G tokens times the G heads of
// the group), walks the keys in tiles of 64 and keeps its output rows in registers, so that a K or V row is fetched once
// per 64 query rows instead of once per token (attention_kernel reads each key's row with one lane, 16 bytes at a time, for
// every token: 370 + 38 us with the merge at 512 tokens of 32 heads of 128, against 136 here).  f32 throughout, as there: the products are
// bound by the FMA pipe and by shared memory (4 x 4 scores and 4 x HD / 16 outputs per thread).  K and V share one
// buffer, which leaves room for two CTAs per SM: one loads while the other multiplies.  The weighted sum of V is added up
// in ATTN_SPLITS shares of the keys and the shares then, as there: one chain over all keys was 2.7 times as far from 64 bits at
// 512 keys, and more with each key.
// ---------------------------------------------------------------------------
constexpr int AP_ROWS = 64, AP_KEYS = 64, AP_PP = AP_KEYS + 4;
template <int HD>
constexpr size_t attention_prompt_smem() { return ((size_t)(AP_ROWS + AP_KEYS) * (HD + 4) + (size_t)AP_ROWS * (AP_PP + 3)) * sizeof(float); }

template <int HD>
__global__ void __launch_bounds__(256, 2) attention_prompt_kernel(const float *__restrict__ qkv, const __half *__restrict__ kc,
                                                                  const __half *__restrict__ vc, float *__restrict__ out,
                                                                  const int *__restrict__ pos, int T, int H, int KV, float scale,
                                                                  int max_ctx) {
    constexpr int PITCH = HD + 4, NV = HD / 64;   // NV: float4 of an output row per thread
    extern __shared__ __align__(16) float ap_s[];
    float *qs = ap_s, *kv = qs + AP_ROWS * PITCH, *ps = kv + AP_KEYS * PITCH;
    // per row, written by the first of its sixteen threads (registers are short): the keys it sees; the sum of weights of
    // the shares that are complete; what the maximum has taken from those since
    float *l_s = ps + AP_ROWS * AP_PP, *since_s = l_s + AP_ROWS;
    int *nk_s = reinterpret_cast<int *>(since_s + AP_ROWS);
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    const int G = H / KV, TQ = AP_ROWS / G;
    const int t0 = (int)(gridDim.x - 1 - blockIdx.x) * TQ, kvh = blockIdx.y;   // the tiles with the most keys first
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int p0 = *pos, ld = (H + 2 * KV) * HD;
    // row r of the tile: token t0 + r / G, head kvh * G + r % G; rows past the last token read zeros and are not stored
    for (int i = tid; i < AP_ROWS * (HD / 4); i += 256) {
        const int r = i / (HD / 4), c = i % (HD / 4), t = t0 + r / G;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < TQ * G && t < T) v = *reinterpret_cast<const float4 *>(qkv + (size_t)t * ld + (size_t)(kvh * G + r % G) * HD + 4 * c);
        *reinterpret_cast<float4 *>(qs + r * PITCH + 4 * c) = v;
    }
    if (tid < AP_ROWS) {
        nk_s[tid] = min(p0 + t0 + tid / G + 1, max_ctx);
        l_s[tid] = 0.f;
        since_s[tid] = 1.f;
    }
    // acc: weighted sum of V of the complete shares, for the maximum at that time; as, ls: of the current one, with its sum
    // of weights, for the maximum m
    float m[4], ls[4], acc[4][NV][4], as[4][NV][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -CUDART_INF_F;
        ls[i] = 0.f;
#pragma unroll
        for (int h = 0; h < NV; ++h)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][h][j] = as[i][h][j] = 0.f;
    }
    const int kmax = min(p0 + min(t0 + TQ, T), max_ctx);     // keys any row of the tile sees
    const int share = ((kmax + AP_KEYS - 1) / AP_KEYS + ATTN_SPLITS - 1) / ATTN_SPLITS * AP_KEYS;   // keys of a share: whole tiles
    int share_end = share;
    const int first_seen = min(p0 + t0 + 1, max_ctx);        // keys every row of the tile sees
    auto load = [&](const __half *src, int k0) {
        for (int i = tid; i < AP_KEYS * (HD / 8); i += 256) {
            const int r = i / (HD / 8), c = i % (HD / 8);
            uint4 u = make_uint4(0u, 0u, 0u, 0u);
            if (k0 + r < kmax) u = *reinterpret_cast<const uint4 *>(src + ((size_t)(k0 + r) * KV + kvh) * HD + 8 * c);
            const __half2 *hp = reinterpret_cast<const __half2 *>(&u);
            const float2 a = __half22float2(hp[0]), b = __half22float2(hp[1]), d = __half22float2(hp[2]), e = __half22float2(hp[3]);
            float4 *dst = reinterpret_cast<float4 *>(kv + r * PITCH + 8 * c);
            dst[0] = make_float4(a.x, a.y, b.x, b.y);
            dst[1] = make_float4(d.x, d.y, e.x, e.y);
        }
    };
    for (int k0 = 0; k0 < kmax; k0 += AP_KEYS) {
        __syncthreads();                          // the buffer's last readers are done
        load(kc, k0);
        __syncthreads();
        // scores of rows 4 ty + i against keys k0 + tx + 16 j
        float s[4][4] = {};
#pragma unroll 4
        for (int d = 0; d < HD; d += 4) {
            float4 q[4], k[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const float4 *>(qs + (4 * ty + i) * PITCH + d);
#pragma unroll
            for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const float4 *>(kv + (tx + 16 * j) * PITCH + d);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    s[i][j] = fmaf(q[i].x, k[j].x, s[i][j]);
                    s[i][j] = fmaf(q[i].y, k[j].y, s[i][j]);
                    s[i][j] = fmaf(q[i].z, k[j].z, s[i][j]);
                    s[i][j] = fmaf(q[i].w, k[j].w, s[i][j]);
                }
        }
        __syncthreads();
        load(vc, k0);
        // running-maximum softmax; a row's sixteen threads are half a warp
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int nk = nk_s[4 * ty + i];
            float cm = -CUDART_INF_F;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[i][j] = k0 + tx + 16 * j < nk ? s[i][j] * scale : -CUDART_INF_F;
                cm = fmaxf(cm, s[i][j]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
            const float mn = fmaxf(m[i], cm);     // finite from the first tile on: every row sees key 0
            const float corr = expf(m[i] - mn);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float pr = k0 + tx + 16 * j < nk ? expf(s[i][j] - mn) : 0.f;
                ps[(4 * ty + i) * AP_PP + tx + 16 * j] = pr;
                sum += pr;
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            ls[i] = ls[i] * corr + sum;
            if (tx == 0) since_s[4 * ty + i] *= corr;
            m[i] = mn;
#pragma unroll
            for (int h = 0; h < NV; ++h)
#pragma unroll
                for (int j = 0; j < 4; ++j) as[i][h][j] *= corr;
        }
        __syncthreads();
        // Outputs of rows 4 ty + i, dimensions 64 h + 4 tx ..  In a tile with keys that some row does not see (masked) such a
        // key's V does not enter the row at all: its weight is zero, but zero times an infinity is not.
        auto weigh = [&](auto form) {
            constexpr bool masked = decltype(form)::value;
            int seen[4];                          // keys of this tile that row 4 ty + i sees
#pragma unroll
            for (int i = 0; i < 4; ++i) seen[i] = masked ? nk_s[4 * ty + i] - k0 : AP_KEYS;
#pragma unroll 2
            for (int k = 0; k < AP_KEYS; k += 4) {
                float4 pr[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) pr[i] = *reinterpret_cast<const float4 *>(ps + (4 * ty + i) * AP_PP + k);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
#pragma unroll
                    for (int h = 0; h < NV; ++h) {
                        const float4 v = *reinterpret_cast<const float4 *>(kv + (k + e) * PITCH + 64 * h + 4 * tx);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            if (masked && k + e >= seen[i]) continue;
                            const float pe = e == 0 ? pr[i].x : e == 1 ? pr[i].y : e == 2 ? pr[i].z : pr[i].w;
                            as[i][h][0] = fmaf(pe, v.x, as[i][h][0]);
                            as[i][h][1] = fmaf(pe, v.y, as[i][h][1]);
                            as[i][h][2] = fmaf(pe, v.z, as[i][h][2]);
                            as[i][h][3] = fmaf(pe, v.w, as[i][h][3]);
                        }
                    }
                }
            }
        };
        if (k0 + AP_KEYS > first_seen) weigh(std::true_type()); else weigh(std::false_type());
        if (k0 + AP_KEYS >= share_end || k0 + AP_KEYS >= kmax) {
            share_end += share;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float since = since_s[4 * ty + i];
#pragma unroll
                for (int h = 0; h < NV; ++h)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        acc[i][h][j] = fmaf(acc[i][h][j], since, as[i][h][j]);
                        as[i][h][j] = 0.f;
                    }
                __syncwarp();                     // all sixteen have read
                if (tx == 0) {
                    l_s[4 * ty + i] = fmaf(l_s[4 * ty + i], since, ls[i]);
                    since_s[4 * ty + i] = 1.f;
                }
                ls[i] = 0.f;
            }
            __syncwarp();
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = 4 * ty + i, t = t0 + r / G;
        if (r >= TQ * G || t >= T) continue;
        const float inv = 1.0f / l_s[r];
#pragma unroll
        for (int h = 0; h < NV; ++h)
            *reinterpret_cast<float4 *>(out + ((size_t)t * H + kvh * G + r % G) * HD + 64 * h + 4 * tx) =
                make_float4(acc[i][h][0] * inv, acc[i][h][1] * inv, acc[i][h][2] * inv, acc[i][h][3] * inv);
    }
}

// arg-max of a row, lowest index on ties (greedy sampling); one CTA.  Ends the step: the position moves on by `by`.
__global__ void __launch_bounds__(1024) argmax_kernel(const float *__restrict__ v, int n, int32_t *__restrict__ out,
                                                      int *pos, int by) {
    __shared__ float bv[32];
    __shared__ int bi[32];
    pdl_wait_prior_grid();
    pdl_launch_dependents();
    float best = -CUDART_INF_F;
    int idx = 0x7fffffff;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float x = v[i];
        if (x > best || (x == best && i < idx)) { best = x; idx = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ob > best || (ob == best && oi < idx)) { best = ob; idx = oi; }
    }
    if ((threadIdx.x & 31) == 0) { bv[threadIdx.x >> 5] = best; bi[threadIdx.x >> 5] = idx; }
    __syncthreads();
    if (threadIdx.x < 32) {
        best = bv[threadIdx.x]; idx = bi[threadIdx.x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
            if (ob > best || (ob == best && oi < idx)) { best = ob; idx = oi; }
        }
        if (threadIdx.x == 0) {
            *out = idx == 0x7fffffff ? 0 : idx;
            *pos += by;
        }
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
int launch_rmsnorm_rows(float *y, const float *x, const float *w, int S, int D, float eps, cudaStream_t st) {
    if (!y || !x || !w || S <= 0 || D <= 0 || D % 4) return ZMOE_ERR_ARG;
    count_launches(1);
    return cu(launch_pdl(rmsnorm_kernel, dim3(S), dim3(256), 0, st, y, x, w, D, eps));
}

int launch_quantize_q8_0(const float *x, int ldx, int8_t *q, float *d, int rows, int I, cudaStream_t st) {
    const long blocks = (long)rows * (I / 32);
    long grid = (blocks + 7) / 8;
    const long cap = 8L * device_sm_count();
    if (grid > cap) grid = cap;
    if (grid < 1) grid = 1;
    count_launches(1);
    return cu(launch_pdl(quantize_q8_0_kernel, dim3((unsigned)grid), dim3(256), 0, st, x, ldx, q, d, rows, I));
}

template <int BM, int BN>
int launch_q8_0_mma(float *y, int ldy, const void *w, const int8_t *xq, const float *xd, int S, int I, int O, int accumulate,
                    cudaStream_t st) {
    const int lacking = (BN - S % BN) % BN;   // rows of the last tile past the batch
    auto fn = lacking > BN / 8 ? q8_0_mma_kernel<BM, BN, true> : q8_0_mma_kernel<BM, BN, false>;
    const size_t smem = (size_t)MQ_NST * mq_stage_bytes<BM, BN>();
    if (raise_dynamic_smem(reinterpret_cast<const void *>(fn), smem) != ZMOE_OK) return ZMOE_ERR_CUDA;
    count_launches(1);
    return cu(launch_pdl(fn, dim3((O + BM - 1) / BM, (S + BN - 1) / BN), dim3(128), smem, st, y, ldy,
                         static_cast<const uint8_t *>(w), xq, xd, S, I, O, accumulate));
}

constexpr int MM_SC = 8;   // activation rows per pass over the weights
int launch_q8_0_mm(float *y, int ldy, const void *w, const int8_t *xq, const float *xd, int S, int I, int O, int accumulate,
                   cudaStream_t st) {
    const int nb = I / 32, rb = nb * 34, rbs = (rb + 32 + 15) & ~15;
    const size_t smem = (size_t)MM_SC * I + (size_t)MM_SC * nb * 4 + (size_t)MM_WARPS * rbs;
    if (smem > 200 * 1024) return ZMOE_ERR_SHAPE;
    if (S > MM_SC && nb % MQ_KB == 0) {
        // more than one pass of the kernel below, and rows that are whole stages (multiples of 272 bytes, so that every
        // copy starts on a 16-byte boundary).  Small tiles where large ones would leave most of the chip idle.
        const long big = (long)((O + 63) / 64) * ((S + 63) / 64);
        return big >= device_sm_count()
                   ? launch_q8_0_mma<64, 64>(y, ldy, w, xq, xd, S, I, O, accumulate, st)
                   : launch_q8_0_mma<32, 32>(y, ldy, w, xq, xd, S, I, O, accumulate, st);
    }
    // one row (a decode step): an instantiation without the other rows' accumulators and buffers, eight CTAs to an SM
    auto fn = S == 1 ? q8_0_matmul_kernel<1> : q8_0_matmul_kernel<MM_SC>;
    const size_t need = S == 1 ? (size_t)I + (((size_t)nb * 4 + 15) & ~(size_t)15) + (size_t)MM_WARPS * rbs : smem;
    if (need > 48 * 1024 && raise_dynamic_smem(reinterpret_cast<const void *>(fn), need) != ZMOE_OK) return ZMOE_ERR_CUDA;
    long grid = ((long)O + MM_WARPS - 1) / MM_WARPS;
    const long cap = (S == 1 ? 8L : 4L) * device_sm_count();
    if (grid > cap) grid = cap;
    count_launches(1);
    return cu(launch_pdl(fn, dim3((unsigned)grid), dim3(32 * MM_WARPS), need, st, y, ldy, static_cast<const uint8_t *>(w),
                         (size_t)O * rb, xq, xd, S, I, O, accumulate));
}

template <int HD>
int launch_attention_prompt(const float *qkv, const __half *kc, const __half *vc, float *out, const int *pos, int T, int H, int KV,
                            float scale, int max_ctx, cudaStream_t st) {
    const int TQ = AP_ROWS / (H / KV);
    auto fn = attention_prompt_kernel<HD>;
    if (raise_dynamic_smem(reinterpret_cast<const void *>(fn), attention_prompt_smem<HD>()) != ZMOE_OK) return ZMOE_ERR_CUDA;
    count_launches(1);
    return cu(launch_pdl(fn, dim3((T + TQ - 1) / TQ, KV), dim3(256), attention_prompt_smem<HD>(), st, qkv, kc, vc, out, pos, T, H, KV,
                         scale, max_ctx));
}

// CTAs of the query tiles of T tokens; 0 where the keys are split instead: too few for half of the chip
int query_tiles(int T, int H, int KV) {
    const int TQ = AP_ROWS / (H / KV), n = (T + TQ - 1) / TQ * KV;
    return n >= device_sm_count() / 2 ? n : 0;
}

// Where the query tiles are about one per SM they must not be placed while the six-head form of RoPE still runs: all of that grid is resident at once, so its
// dependants may come at once too, and find room for two beside each other on some SMs while others get none.  (A head per CTA is too many CTAs for
// that; the tiles then came as the last of them left.)  A prompt step of two layers of 2048 / 768, us, tiles early / late, by tiles on 148 SMs: 32 heads
// on 4 of 128 76 590 / 590, 100 751 / 720, 120 832 / 789, 148 964 / 914, 156 1009 / 961, 176 1109 / 1094, 188 1134 / 1135, 192 817 / 827, 228 908 /
// 896, 300 1149 / 1173; 64 on 8 80 562 / 578, 96 595 / 607, 104 623 / 600, 144 724 / 701, 176 783 / 770, 184 769 / 800; 32 on 8 104 763 / 726, 136 932 / 886,
// 176 1108 / 1100; 16 on 2 100 676 / 665, 126 825 / 742, 176 1038 / 957; of 64 16 on 16 112 635 / 615.  With split keys early: 64 on 8, 40 tokens 425 / 454.
bool rope_holds_attention(int tiles) {
    const int n = device_sm_count();
    return 3 * tiles >= 2 * n && 5 * tiles <= 6 * n;
}

// Attention of T tokens, its rows quantised to Q8_0 (aq, ad): by query tiles where those are enough CTAs for half of the chip (a tile walks all keys on its
// own, and the number of earlier positions is not known here); below that, keys split over CTAs token by token.
template <int HD>
int launch_attention(const float *qkv, const __half *kc, const __half *vc, float *part, float *out, const int *pos, int T, int H,
                     int KV, float scale, int max_ctx, int8_t *aq, float *ad, cudaStream_t st) {
    const int G = H / KV;
    if (query_tiles(T, H, KV)) {
        const int rc = launch_attention_prompt<HD>(qkv, kc, vc, out, pos, T, H, KV, scale, max_ctx, st);
        return rc ? rc : launch_quantize_q8_0(out, H * HD, aq, ad, T, H * HD, st);
    }
    count_launches(2);
    int rc = cu(launch_pdl(attention_kernel<HD>, dim3(T, KV, ATTN_SPLITS), dim3(32 * G), (size_t)G * HD * sizeof(float), st, qkv,
                           kc, vc, part, pos, H, KV, scale, max_ctx));
    if (!rc) rc = cu(launch_pdl(attention_merge_q8_0_kernel<HD>, dim3((T * H + 7) / 8), dim3(256), 0, st, (const float *)part, aq,
                                ad, T * H));
    return rc;
}

// per-device scratch of the handle-free Q8_0 entry: quantised activations
struct Q8Scratch {
    int8_t *q = nullptr;
    float *d = nullptr;
    size_t cap = 0;   // elements
};
Q8Scratch g_q8[64];
std::mutex g_q8_mu;

}  // namespace

// ---------------------------------------------------------------------------
// the decoder
// ---------------------------------------------------------------------------
struct zmoe_decoder {
    zmoe_decoder_desc d;
    std::vector<const float *> attn_norm, ffn_norm;
    std::vector<const void *> wqkv, wo;
    std::vector<zmoe_layer *> moe;
    int qkv_cols = 0;
    float *h = nullptr, *xn = nullptr, *qkv = nullptr, *ao = nullptr, *logits = nullptr, *apart = nullptr;
    int8_t *aq = nullptr;
    float *ad = nullptr;
    __half *kc = nullptr, *vc = nullptr;     // [layers][max_ctx][KV * hd]
    int *pos = nullptr;                      // followed by the step kernel's synchronisation words: a reset clears both
    size_t pos_words = 1;
    int32_t *next = nullptr;
    DecoderStep *step = nullptr;             // one-token steps in one kernel, where the shapes allow it
};

extern "C" {

void launch_rmsnorm(float *y, const float *x, const float *w, int S, int D, float eps) {
    set_last_status(launch_rmsnorm_rows(y, x, w, S, D, eps, nullptr));
}

void launch_q8_0_matmul_stream(float *y, const float *x, const void *weights, int S, int I, int O, void *stream) {
    if (!y || !x || !weights || S <= 0 || I <= 0 || O <= 0) { set_last_status(ZMOE_ERR_ARG); return; }
    if (I % 32) { set_last_status(ZMOE_ERR_SHAPE); return; }
    if (reinterpret_cast<size_t>(weights) & 15) { set_last_status(ZMOE_ERR_ALIGN); return; }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { set_last_status(ZMOE_ERR_CUDA); return; }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // the scratch stays locked from sizing to enqueue; it is reallocated only after the device has drained
    std::lock_guard<std::mutex> lock(g_q8_mu);
    Q8Scratch &s = g_q8[dev];
    const size_t need = (size_t)S * I;
    if (need > s.cap) {
        if (s.q) { cudaDeviceSynchronize(); cudaFree(s.q); cudaFree(s.d); s.q = nullptr; s.d = nullptr; s.cap = 0; }
        if (cudaMalloc(reinterpret_cast<void **>(&s.q), need) != cudaSuccess ||
            cudaMalloc(reinterpret_cast<void **>(&s.d), (need / 32) * sizeof(float)) != cudaSuccess) {
            set_last_status(ZMOE_ERR_CUDA);
            return;
        }
        s.cap = need;
    }
    int rc = launch_quantize_q8_0(x, I, s.q, s.d, S, I, st);
    if (!rc) rc = launch_q8_0_mm(y, O, weights, s.q, s.d, S, I, O, 0, st);
    set_last_status(rc);
}

void launch_q8_0_matmul(float *y, const float *x, const void *weights, int S, int I, int O) {
    launch_q8_0_matmul_stream(y, x, weights, S, I, O, nullptr);
}

void zmoe_decoder_destroy(zmoe_decoder *dec) {
    if (!dec) return;
    decoder_step_destroy(dec->step);
    cudaFree(dec->h); cudaFree(dec->xn); cudaFree(dec->qkv); cudaFree(dec->ao); cudaFree(dec->logits); cudaFree(dec->apart);
    cudaFree(dec->aq); cudaFree(dec->ad); cudaFree(dec->kc); cudaFree(dec->vc); cudaFree(dec->pos); cudaFree(dec->next);
    delete dec;
}

int zmoe_decoder_create(const zmoe_decoder_desc *desc, zmoe_decoder **out) {
    if (!desc || !out) return ZMOE_ERR_ARG;
    const zmoe_decoder_desc &d = *desc;
    if (d.n_layers <= 0 || d.d_model <= 0 || d.n_heads <= 0 || d.n_kv_heads <= 0 || d.vocab <= 0 || d.max_ctx <= 0 ||
        d.max_tokens <= 0 || !d.attn_norm_w || !d.wqkv || !d.wo || !d.ffn_norm_w || !d.moe || !d.tok_embd ||
        !d.out_norm_w || !d.lm_head)
        return ZMOE_ERR_ARG;
    if ((d.head_dim != 64 && d.head_dim != 128) || d.n_heads % d.n_kv_heads || d.n_heads / d.n_kv_heads > 32 ||
        d.d_model % 32 || (d.n_heads * d.head_dim) % 32)
        return ZMOE_ERR_SHAPE;
    zmoe_decoder *dec = new (std::nothrow) zmoe_decoder();
    if (!dec) return ZMOE_ERR_ARG;
    dec->d = d;
    for (int l = 0; l < d.n_layers; ++l) {
        if (!d.attn_norm_w[l] || !d.wqkv[l] || !d.wo[l] || !d.ffn_norm_w[l] || !d.moe[l]) {
            delete dec;
            return ZMOE_ERR_ARG;
        }
        dec->attn_norm.push_back(d.attn_norm_w[l]);
        dec->ffn_norm.push_back(d.ffn_norm_w[l]);
        dec->wqkv.push_back(d.wqkv[l]);
        dec->wo.push_back(d.wo[l]);
        dec->moe.push_back(d.moe[l]);
    }
    dec->qkv_cols = (d.n_heads + 2 * d.n_kv_heads) * d.head_dim;
    const size_t T = d.max_tokens, D = d.d_model, QO = (size_t)d.n_heads * d.head_dim;
    const size_t widest = D > QO ? D : QO;
    const size_t kv = (size_t)d.n_layers * d.max_ctx * d.n_kv_heads * d.head_dim;
    auto A = [](auto **p, size_t n) { return cudaMalloc(reinterpret_cast<void **>(p), (n ? n : 1) * sizeof(**p)) != cudaSuccess; };
    int bad = 0;
    bad |= A(&dec->h, T * D); bad |= A(&dec->xn, T * D); bad |= A(&dec->qkv, T * dec->qkv_cols); bad |= A(&dec->ao, T * QO);
    bad |= A(&dec->logits, (size_t)d.vocab);
    bad |= A(&dec->apart, T * d.n_heads * ATTN_SPLITS * (d.head_dim + 2));
    bad |= A(&dec->aq, T * widest); bad |= A(&dec->ad, T * widest / 32);
    bad |= A(&dec->kc, kv); bad |= A(&dec->vc, kv);
    dec->pos_words = 2 + (size_t)decoder_step_sync_words(d.n_kv_heads);
    bad |= A(&dec->pos, dec->pos_words); bad |= A(&dec->next, 1);
    if (!bad) bad |= cudaMemset(dec->pos, 0, dec->pos_words * sizeof(int)) != cudaSuccess || cudaMemset(dec->next, 0, sizeof(int32_t)) != cudaSuccess;
    if (bad) {
        zmoe_decoder_destroy(dec);
        return ZMOE_ERR_CUDA;
    }
    DecoderStepDesc sd = {};
    sd.n_layers = d.n_layers;
    sd.attn_norm = dec->attn_norm.data(); sd.ffn_norm = dec->ffn_norm.data(); sd.wqkv = dec->wqkv.data(); sd.wo = dec->wo.data();
    sd.moe = dec->moe.data();
    sd.embd = d.tok_embd; sd.head = d.lm_head; sd.out_norm = d.out_norm_w;
    sd.D = d.d_model; sd.H = d.n_heads; sd.KV = d.n_kv_heads; sd.HD = d.head_dim; sd.vocab = d.vocab; sd.max_ctx = d.max_ctx;
    sd.splits = ATTN_SPLITS;
    sd.eps = d.rms_eps; sd.theta_scale = powf(d.rope_theta, -2.0f / (float)d.head_dim); sd.scale = 1.0f / sqrtf((float)d.head_dim);
    sd.h = dec->h; sd.xn = dec->xn; sd.qkv = dec->qkv; sd.part = dec->apart; sd.logits = dec->logits; sd.aq = dec->aq; sd.ad = dec->ad;
    sd.kc = dec->kc; sd.vc = dec->vc; sd.pos = dec->pos; sd.next = dec->next;
    sd.sync = reinterpret_cast<unsigned *>(dec->pos) + 2;
    dec->step = decoder_step_create(sd);     // null: the separate launches
    *out = dec;
    return ZMOE_OK;
}

int zmoe_decoder_reset(zmoe_decoder *dec, void *stream) {
    if (!dec) return ZMOE_ERR_ARG;
    return cu(cudaMemsetAsync(dec->pos, 0, dec->pos_words * sizeof(int), static_cast<cudaStream_t>(stream)));
}

int zmoe_decoder_step(zmoe_decoder *dec, const int32_t *tokens_dev, int T, void *stream) {
    if (!dec || T <= 0) return ZMOE_ERR_ARG;
    const zmoe_decoder_desc &d = dec->d;
    if (T > d.max_tokens) return ZMOE_ERR_CAPACITY;
    if (!tokens_dev) {
        if (T != 1) return ZMOE_ERR_ARG;
        tokens_dev = dec->next;             // the token the previous step produced
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (T == 1 && dec->step) {
        const int one = decoder_step_launch(dec->step, tokens_dev, st);
        if (one != ZMOE_ERR_STATE) return one;
    }
    const int D = d.d_model, H = d.n_heads, KV = d.n_kv_heads, hd = d.head_dim, QO = H * hd;
    const size_t kv_layer = (size_t)d.max_ctx * KV * hd;
    const float scale = 1.0f / sqrtf((float)hd);
    const float theta_scale = powf(d.rope_theta, -2.0f / (float)hd);
    int rc = cu(launch_pdl(embed_q8_0_kernel, dim3(T), dim3(256), 0, st, tokens_dev, static_cast<const uint8_t *>(d.tok_embd),
                           dec->h, D, d.vocab));
    count_launches(1);
    for (int l = 0; l < d.n_layers && !rc; ++l) {
        // ---- attention block: h += Wo . attention(rope(Wqkv . rmsnorm(h))) ----
        rc = cu(launch_pdl(rmsnorm_q8_0_kernel, dim3(T), dim3(256), 0, st, dec->aq, dec->ad, (const float *)dec->h,
                           (const float *)dec->attn_norm[l], D, d.rms_eps));
        count_launches(1);
        if (!rc) rc = launch_q8_0_mm(dec->qkv, dec->qkv_cols, dec->wqkv[l], dec->aq, dec->ad, T, D, dec->qkv_cols, 0, st);
        const bool six = T >= ROPE_TOKENS;
        if (!rc) rc = cu(launch_pdl(six ? rope_kv_kernel<6> : rope_kv_kernel<1>, dim3(T, six ? (H + KV + 5) / 6 : H + KV), dim3(hd / 2), 0, st, dec->qkv,
                                    dec->kc + l * kv_layer, dec->vc + l * kv_layer, (const int *)dec->pos, H, KV, hd, theta_scale, d.max_ctx,
                                    six && rope_holds_attention(query_tiles(T, H, KV)) ? 1 : 0));
        if (!rc) {
            const __half *kl = dec->kc + l * kv_layer, *vl = dec->vc + l * kv_layer;
            rc = hd == 128 ? launch_attention<128>(dec->qkv, kl, vl, dec->apart, dec->ao, dec->pos, T, H, KV, scale, d.max_ctx, dec->aq, dec->ad, st)
                           : launch_attention<64>(dec->qkv, kl, vl, dec->apart, dec->ao, dec->pos, T, H, KV, scale, d.max_ctx, dec->aq, dec->ad, st);
        }
        count_launches(1);
        if (!rc) rc = launch_q8_0_mm(dec->h, D, dec->wo[l], dec->aq, dec->ad, T, QO, D, 1, st);
        // ---- MoE block: h += MoE(rmsnorm(h)) ----
        if (!rc) rc = launch_rmsnorm_rows(dec->xn, dec->h, dec->ffn_norm[l], T, D, d.rms_eps, st);
        if (!rc) rc = layer_forward(dec->moe[l], dec->xn, dec->h, T, 1, stream);
    }
    // ---- output head on the last token, greedy sampling ----
    if (!rc) {
        rc = cu(launch_pdl(rmsnorm_q8_0_kernel, dim3(1), dim3(256), 0, st, dec->aq, dec->ad,
                           (const float *)(dec->h + (size_t)(T - 1) * D), (const float *)d.out_norm_w, D, d.rms_eps));
        count_launches(1);
    }
    if (!rc) rc = launch_q8_0_mm(dec->logits, d.vocab, d.lm_head, dec->aq, dec->ad, 1, D, d.vocab, 0, st);
    if (!rc) rc = cu(launch_pdl(argmax_kernel, dim3(1), dim3(1024), 0, st, (const float *)dec->logits, d.vocab, dec->next, dec->pos, T));
    count_launches(1);
    return rc;
}

int zmoe_attention_rows(const float *qkv_dev, const void *k_dev, const void *v_dev, float *out_dev, const int *pos_dev, int T, int H,
                        int KV, int head_dim, int max_ctx, void *stream) {
    if (!qkv_dev || !k_dev || !v_dev || !out_dev || !pos_dev || T <= 0 || H <= 0 || KV <= 0 || max_ctx <= 0) return ZMOE_ERR_ARG;
    if ((head_dim != 64 && head_dim != 128) || H % KV || H / KV > 32) return ZMOE_ERR_SHAPE;
    const __half *k = static_cast<const __half *>(k_dev), *v = static_cast<const __half *>(v_dev);
    const float scale = 1.0f / sqrtf((float)head_dim);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return head_dim == 128 ? launch_attention_prompt<128>(qkv_dev, k, v, out_dev, pos_dev, T, H, KV, scale, max_ctx, st)
                           : launch_attention_prompt<64>(qkv_dev, k, v, out_dev, pos_dev, T, H, KV, scale, max_ctx, st);
}

int zmoe_decoder_read(zmoe_decoder *dec, int32_t *next_token_host, int32_t *pos_host, float *logits_host, int n_logits) {
    if (!dec) return ZMOE_ERR_ARG;
    int rc = 0;
    if (next_token_host) rc |= cu(cudaMemcpy(next_token_host, dec->next, sizeof(int32_t), cudaMemcpyDeviceToHost));
    if (pos_host) rc |= cu(cudaMemcpy(pos_host, dec->pos, sizeof(int32_t), cudaMemcpyDeviceToHost));
    if (logits_host && n_logits > 0)
        rc |= cu(cudaMemcpy(logits_host, dec->logits, (size_t)(n_logits < dec->d.vocab ? n_logits : dec->d.vocab) * sizeof(float),
                            cudaMemcpyDeviceToHost));
    return rc ? ZMOE_ERR_CUDA : ZMOE_OK;
}

}  // extern "C"
