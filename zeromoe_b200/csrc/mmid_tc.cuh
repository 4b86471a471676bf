// mmid_tc.cuh -- the MUL_MAT_ID kernel for experts that hold a few to a few dozen pairs: quantised expert rows against Q8_K
// activations on the 5th-generation tensor cores, in integers (tcgen05.mma kind::i8, s32 accumulate).
//
// Same job and same arithmetic contract as mmid2.cuh (replaces reference core/gpu_expert_executor.cpp:358-387,512-513 and
// kernels/quant/kquant_matmul.cu:647-700): the sums of a super-block are exact integers, the f32 assembly multiplies them by
// d_w * d_x and adds super-blocks in ascending order, in chains of four whose sums are added up in turn (one chain over a row of
// 7168 left SwiGLU values 1.43e-7 of their size from 64 bits where the slices and lanes of the other kernels left 1.11e-7; chains of four
// 1.03e-7).  A pair's result depends on its own row and weights alone,
// not on which other pairs share its expert.
//
// An item is (expert, 128 weight rows -- 64 gate rows and the same 64 up rows in DUAL mode --, up to BN pairs).  Per
// super-block of 256 k one thread converts half a row to int8 and stores it as its lane of the A operand in tensor memory:
//   Q2_K     scale * quant (at most 45) as unsigned bytes; the mins meet the group sums of the activations in one
//            kind::f16 instruction on exact small integers, in an accumulator of its own
//   Q3_K     128 - scale * (quant - 4) as unsigned bytes (0..252 for scales of -32..31: one multiply-add per four weights, no byte
//            borrows from the next); 128 times the sum of the activations is taken off afterwards
//   IQ2_XXS  sign * magnitude * (2 ls + 1) = 128 hi + lo, two planes of signed bytes looked up by byte permutes
// Warps 0-3 drain: they read a finished super-block's sums from tensor memory and add them, scaled, to the item's f32 results
// in registers.  Warps 4-19 convert, in four groups that take half super-blocks in turn; warp 20 brings raw blocks (tiled copies, no
// multicast), warp 21 issues the MMAs, warps 22-23 bring the activations of alternate super-blocks: 16-byte asynchronous copies of the
// pairs' packed rows, wherever these lie, into the swizzled layout that the MMA reads (the rows need no gather of their own).
// What bounds it: not the tensor core (7 %) and not HBM but the converters' and the drain's issue slots (63 %) and the way there and back of
// a super-block (operand store, barrier, MMAs, commit, drain, with up to four on their way).  Its cost hardly
// grows with the pairs of an expert, that of mmid2.cuh with every eight of them.  Layer times beside the rule that chooses (api.cu,
// takes_tc).  Two waits of one warp in one instruction (lanes polling different barriers) do not work: the poll goes by one lane's barrier.
// Accumulators rotate by super-block, an operand slot holds one.  The registers of a launch (80 a thread) are
// dealt out by role: the drain keeps an item's results in them.
// Every wait is bounded; on expiry the warp raises the error flag and leaves, and the tensor memory is always released.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "dequant_f16.cuh"
#include "mmid.cuh"

namespace zmoe {

constexpr int TC_THREADS = 768;
constexpr int TC_CONV0 = 4, TC_TMA = 20, TC_MMA = 21, TC_LOAD0 = 22;   // first converter, weight copies, MMA issue, first activation loader
// registers per thread: of the launch, and of the warpgroups' roles, which add up to six times the launch's
constexpr int TC_REGS = 80, TC_REGS_DRAIN = 136, TC_REGS_CONV = 72, TC_REGS_MISC = 56;
static_assert(TC_REGS_DRAIN + 4 * TC_REGS_CONV + TC_REGS_MISC == 6 * TC_REGS, "registers");
constexpr int TC_NB = 4;            // activation slots (one super-block each)
constexpr int TC_RING = 8;          // super-blocks whose barriers, and scales that travel beside the operands, are kept apart
constexpr int TC_ITEMS = 4;         // items resolved ahead
constexpr int TC_MAXRAW = 8;        // raw stages at most
constexpr int TC_IQ2_COPIES = 8;    // copies of the IQ2_XXS tables: four lanes share one

// kPlanes: byte planes of the A operand; kMin: the format has mins; kAcc: tensor-memory columns for accumulators; kSlots: operand slots, a
// super-block each.  kAcc + (64 * kPlanes + 8 * kMin) * kSlots columns of 512.
// (Q4_K was built too, as two planes of quant & 3 and quant >> 2 times the scale with 48 pairs per item: 2048 / 768 with 64 tokens 198 us
// against 134 of mmid2.cuh, 7168 / 2048 1780 against 1056; its scales of 4.5 bits a weight leave the other kernel less to gain from.)
template <int TYPE> struct TcGeom;
template <> struct TcGeom<Q2_K> { static constexpr int kPlanes = 1, kMin = 1, kAcc = 256, kSlots = 3; };
template <> struct TcGeom<Q3_K> { static constexpr int kPlanes = 1, kMin = 0, kAcc = 128, kSlots = 4; };
template <> struct TcGeom<IQ2_XXS> { static constexpr int kPlanes = 2, kMin = 0, kAcc = 256, kSlots = 2; };
constexpr int TC_BN = 32;           // pairs per item at most
constexpr int TC_SETS = 4;          // sets of accumulators: kAcc / ((kPlanes + kMin) * TC_BN)
constexpr int TC_CHAIN = 4;         // super-blocks that one chain of f32 additions takes

struct TcParams {
    int I, O, rb, g_log2;        // k extent, rows per expert, bytes per row, log2 of the rows per group of the weight maps
    int cb_log2, pitch;          // super-blocks per raw chunk (1 or 2); bytes between rows of a chunk in shared memory
    int nraw, bnr;               // raw stages; pairs an activation slot has room for (a multiple of 16, at most TC_BN)
    int mt;                      // pairs per item the plan was built with
    const uint8_t *q8;
    int q8_stride, xdiv;
    float *y;
    int ldy;
    PlanView plan;
    int hdr_items;
    float clamp;
    int clamp_fused;
    int *err, *bad;
    alignas(64) CUtensorMap tm0, tm1;
};

// D[tmem] (+)= A[tmem] * B[smem], 8-bit integers, s32 accumulate; issued by one thread.  A: lane = row, a 32-bit column holds four
// consecutive k, so a k-step of 32 advances the address by 8 columns
__device__ __forceinline__ void umma_i8_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// instruction descriptor, kind::i8: s32 accumulate (bits 4-5 = 2), A unsigned (bits 7-9 = 0) or signed (1), B signed (bits 10-12 = 1)
__host__ __device__ constexpr uint32_t umma_idesc_i8(int M, int N, bool signed_a) {
    return (2u << 4) | ((signed_a ? 1u : 0u) << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// K-major tile of rows of 32 bytes with the 32-byte swizzle: 16-byte half h of row r lies at 32 r + 16 (h ^ (r / 4 % 2));
// 256 bytes between groups of eight rows, swizzle mode 6
__device__ __forceinline__ uint64_t umma_desc_sw32(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(256 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)6 << 61);
}

__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_32xn(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld_32x16(taddr, r); }
__device__ __forceinline__ void tmem_st_32x8(uint32_t taddr, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
                 "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_st_32x4(uint32_t taddr, const uint32_t (&r)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
                 : "memory");
}
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_8(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void tmem_ld_32xn(uint32_t taddr, uint32_t (&r)[8]) { tmem_ld_32x8(taddr, r); }
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void tc_load_3d(uint32_t dst_smem, const void *tmap, int x, int row, int expert, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst_smem), "l"(tmap), "r"(x), "r"(row), "r"(expert), "r"(smem_u32(bar))
        : "memory");
}

// fp16 pair of two small integers in the two halves of x (at most 1023 each)
__device__ __forceinline__ uint32_t small_f16x2(uint32_t x) { return h2_bits(__hsub2(bits_h2(x | 0x64006400u), bits_h2(0x64006400u))); }

// Half N (128 k) of one row's super-block.  blk: shared address of its first byte; uni: the block's offset from a 16-byte boundary is the
// same in all lanes.  load takes what the conversion needs of it, store puts it into the operand slot: 32 columns of four k per plane.
template <int TYPE> struct TcHalf;

// scales[16] @0 (scale | min << 4), qs[64] @16, d @80, dmin @82.  k = 64 (2n + h) + 16 s + i is byte 32n + 16h + i at bit 2s, group 8n + 2s + h
template <> struct TcHalf<Q2_K> {
    uint32_t q[8], s[2], d;
    __device__ __forceinline__ void load(uint32_t blk, int n, bool uni) {
        const uint32_t w = (blk >> 2) & 3u, at = blk - 4 * w + 16 + 32 * n;
        if (!uni) lds_window<8>(at, 4 * w, q);
        else if (w == 0) lds_words<8, 0>(at, q);
        else if (w == 1) lds_words<8, 1>(at, q);
        else if (w == 2) lds_words<8, 2>(at, q);
        else lds_words<8, 3>(at, q);
        s[0] = lds32(blk + 8 * n);
        s[1] = lds32(blk + 8 * n + 4);
        if (n == 0) d = lds32(blk + 80);
    }
    __device__ __forceinline__ void conv(uint32_t (&o)[32]) const {
        const uint32_t sc[2] = {s[0] & 0x0F0F0F0Fu, s[1] & 0x0F0F0F0Fu};
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int sh = 0; sh < 4; ++sh) {
                const int g = 2 * sh + h;
                const uint32_t f = __byte_perm(sc[g >> 2], 0, 0x4440u | (g & 3));
#pragma unroll
                for (int j = 0; j < 4; ++j) o[16 * h + 4 * sh + j] = ((q[4 * h + j] >> (2 * sh)) & 0x03030303u) * f;
            }
    }
    // fp16 mins of groups 8n .. 8n + 7, pairs (0, 2), (1, 3), (4, 6), (5, 7)
    __device__ __forceinline__ void mins(uint32_t (&o)[4]) const {
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            o[2 * w] = small_f16x2((s[w] >> 4) & 0x000F000Fu);
            o[2 * w + 1] = small_f16x2((s[w] >> 12) & 0x000F000Fu);
        }
    }
};

// hmask[32] @0, qs[64] @32, scales[12] @96, d @108; k as for Q2_K, high bit of it: bit 4n + s of hmask byte 16h + i.  With
// m = 32 - scale: byte = m * q + 128 - 4 m = 128 - (scale - 32) * (q - 4)
template <> struct TcHalf<Q3_K> {
    uint32_t q[8], hm[8], m[2], d;
    __device__ __forceinline__ void load(uint32_t blk, int n, bool uni) {
        uint32_t t[3];
        if (uni) {
            const uint32_t off = blk & 15u, base = blk - off;
            lds_window<8>(base, off, hm);
            lds_window<8>(base + 32 + 32 * n, off, q);
            lds_window<3>(base + 96, off, t);
        } else {
            lds32xN_any<2, 8>(blk, hm);
            lds32xN_any<2, 8>(blk + 32 + 32 * n, q);
            lds32xN_any<2, 3>(blk + 96, t);
        }
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const uint32_t s6 = ((t[w] >> (4 * n)) & 0x0F0F0F0Fu) | (((t[2] >> (4 * n + 2 * w)) & 0x03030303u) << 4);
            // 32 - s6 per byte: with bit 7 set the subtraction cannot borrow across bytes
            m[w] = (0xA0A0A0A0u - s6) ^ 0x80808080u;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) hm[i] >>= 4 * n;
        if (n == 0) d = lds16(blk + 108);
    }
    __device__ __forceinline__ void conv(uint32_t (&o)[32]) const {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int sh = 0; sh < 4; ++sh) {
                const int g = 2 * sh + h;
                const int f = sext_byte(m[g >> 2], g & 3);
                const uint32_t c = 0x80808080u - (uint32_t)f * 0x04040404u;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t hb = (sh < 2 ? hm[4 * h + j] << (2 - sh) : hm[4 * h + j] >> (sh - 2)) & 0x04040404u;
                    o[16 * h + 4 * sh + j] = (((q[4 * h + j] >> (2 * sh)) & 0x03030303u) | hb) * (uint32_t)f + c;
                }
            }
    }
};

// d @0, per sub-block of 32 k: four codebook indices (aux0), four 7-bit sign patterns and a four-bit scale ls (aux1).
// tab: 256 words of eight codes (0, 1, 2 for the magnitudes 8, 25, 43, a nibble each), 128 words of eight signs (4 per minus, a
// nibble each), both in TC_IQ2_COPIES copies, then 16 x 16 bytes: lo and -lo, hi and -hi of the three magnitudes times 2 ls + 1
constexpr int TC_IQ2_SIGNS = 256 * TC_IQ2_COPIES * 4, TC_IQ2_MAGS = TC_IQ2_SIGNS + 128 * TC_IQ2_COPIES * 4, TC_IQ2_BYTES = TC_IQ2_MAGS + 256;
template <> struct TcHalf<IQ2_XXS> {
    uint32_t x[8], d;
    __device__ __forceinline__ void load(uint32_t blk, int n, bool uni) {
        const uint32_t at = blk + 2 + 32 * n;
        if (uni) lds_window<8>(at & ~15u, at & 15u, x);
        else lds32xN_any<2, 8>(at, x);
        if (n == 0) d = lds16(blk);
    }
    // both planes, eight columns of each at a time
    __device__ __forceinline__ void store2(uint32_t tab, uint32_t slot) const {
        const uint32_t codes = tab + 4 * (threadIdx.x & (TC_IQ2_COPIES - 1)), signs = codes + TC_IQ2_SIGNS;
#pragma unroll
        for (int ib = 0; ib < 4; ++ib) {
            const uint32_t a0 = x[2 * ib], a1 = x[2 * ib + 1];
            const uint4 mg = lds128(tab + TC_IQ2_MAGS + 16 * (a1 >> 28));
            uint32_t o[8], o2[8];
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                const uint32_t sel = lds32(codes + 4 * TC_IQ2_COPIES * ((a0 >> (8 * l)) & 255u)) ^
                                     lds32(signs + 4 * TC_IQ2_COPIES * ((a1 >> (7 * l)) & 127u));
                o[2 * l] = __byte_perm(mg.x, mg.y, sel);
                o[2 * l + 1] = __byte_perm(mg.x, mg.y, sel >> 16);
                o2[2 * l] = __byte_perm(mg.z, mg.w, sel);
                o2[2 * l + 1] = __byte_perm(mg.z, mg.w, sel >> 16);
            }
            tmem_st_32x8(slot + 8 * ib, o);
            tmem_st_32x8(slot + 64 + 8 * ib, o2);
        }
    }
};
__device__ __forceinline__ void tc_fill_tables(uint32_t tab) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        const uint64_t g = k_iq2xxs_grid[i];
        uint32_t w = 0;
        for (int e = 0; e < 8; ++e) w |= ((uint32_t)(g >> (8 * e + 4)) & 3u) << (4 * e);   // 0x08, 0x19, 0x2b
        for (int c = 0; c < TC_IQ2_COPIES; ++c) sts32(tab + 4 * (i * TC_IQ2_COPIES + c), w);
    }
    for (int i = threadIdx.x; i < 128; i += blockDim.x) {
        uint32_t w = 0;
        for (int e = 0; e < 8; ++e) w |= ((e < 7 ? i >> e : __popc(i)) & 1u) << (4 * e + 2);
        for (int c = 0; c < TC_IQ2_COPIES; ++c) sts32(tab + TC_IQ2_SIGNS + 4 * (i * TC_IQ2_COPIES + c), w);
    }
    for (int i = threadIdx.x; i < 16; i += blockDim.x) {
        uint32_t w[4] = {0, 0, 0, 0};
        for (int m = 0; m < 3; ++m) {
            const int v = (m == 0 ? 8 : m == 1 ? 25 : 43) * (2 * i + 1);
            w[0] |= (uint32_t)(v & 127) << (8 * m);
            w[1] |= ((uint32_t)(-(v & 127)) & 255u) << (8 * m);
            w[2] |= (uint32_t)(v >> 7) << (8 * m);
            w[3] |= ((uint32_t)(-(v >> 7)) & 255u) << (8 * m);
        }
        for (int k = 0; k < 4; ++k) sts32(tab + TC_IQ2_MAGS + 16 * i + 4 * k, w[k]);
    }
}

// the same answer in all lanes: whether a phase is complete
__device__ __forceinline__ bool mbar_test_warp(uint64_t *bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_test_wait(bar, parity)); }

// Barriers.  Super-block j of the CTA's run (counted through its items) uses entry j % TC_RING of two rings:
//   in[j]    everything its MMAs need: eight converter warps, one activation loader, and the four drain warps, which arrive for j
//            when they are through with super-block j - TC_SETS (its accumulators' last use)
//   done[j]  its MMAs have finished (tcgen05.commit): its sums can be drained, its operand and activation slots refilled
// No waiter can be a whole ring behind: each of them arrives on the in[] of a later super-block first.
template <int TYPE, bool DUAL>
__global__ void __launch_bounds__(TC_THREADS, 1) mmid_tc_kernel(const __grid_constant__ TcParams p) {
    using G = TcGeom<TYPE>;
    constexpr int BB = QTraits<TYPE>::kBytes, BN = TC_BN, PL = G::kPlanes, NACC = PL + G::kMin, NA = G::kSlots;
    constexpr int A_COL = G::kAcc, A_COLS = 64 * PL + 8 * G::kMin;   // operand slots
    static_assert(NACC * BN * TC_SETS <= A_COL && A_COL + A_COLS * NA <= 512 && NA < TC_RING - 2 && TC_NB < TC_RING - 2, "tensor memory, rings");
    constexpr int XP = BN + 1;                           // floats per row of the exchange between gate and up rows
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t raw_full[TC_MAXRAW], raw_empty[TC_MAXRAW], in_full[TC_RING], done[TC_RING], item_full[TC_ITEMS],
        item_empty[TC_ITEMS], x_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(16) int s_item[TC_ITEMS][4];    // expert, first row, -, pairs
    __shared__ __align__(16) int s_pair[TC_ITEMS][BN];
    __shared__ uint32_t s_off[2][BN];                    // the loaders' activation rows, in 16 bytes
    __shared__ uint32_t s_meta[TC_RING][128];            // d (and dmin) of the super-block of each row
    __shared__ __align__(16) uint2 s_dx[TC_RING][BN];    // per pair: d of the activations, 128 times their sum (Q3_K)
    __shared__ float s_x[DUAL ? 128 * XP : 1];
    __shared__ int s_item_offs[MMID_PLAN_SMEM + 1], s_active[MMID_PLAN_SMEM], s_aoffs[MMID_PLAN_SMEM], s_antok[MMID_PLAN_SMEM];
    __shared__ __align__(16) uint32_t s_tab[TYPE == IQ2_XXS ? TC_IQ2_BYTES / 4 : 4];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t smem = (smem_u32(smem_raw) + 1023) & ~1023u;
    const uint32_t b_bytes = (uint32_t)p.bnr * 256u;
    const uint32_t bs_base = smem + TC_NB * b_bytes;                       // fp16 group sums of each slot
    const uint32_t raw_base = (bs_base + TC_NB * (uint32_t)p.bnr * 32u + 127) & ~127u;
    const uint32_t raw_bytes = 128u * (uint32_t)p.pitch;
    if (tid == 0) {
        for (int s = 0; s < TC_MAXRAW; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], 16); }
        for (int s = 0; s < TC_RING; ++s) { mbar_init(&in_full[s], 8 + 1 + 4); mbar_init(&done[s], 1); }
        for (int s = 0; s < TC_ITEMS; ++s) { mbar_init(&item_full[s], 1); mbar_init(&item_empty[s], 4 + 1 + 2); }
        mbar_init(&x_bar, 4);
        mbar_init_fence();
    }
    if (warp == 0) tmem_alloc(&tmem_slot, 512);
    if (TYPE == IQ2_XXS) tc_fill_tables(smem_u32(s_tab));

    pdl_wait_prior_grid();
    pdl_launch_dependents();

    const int n_items = p.plan.hdr[p.hdr_items], n_active = p.plan.hdr[0];
    for (int i = tid; i < MMID_PLAN_SMEM && i < p.plan.cap_e; i += blockDim.x) {
        s_item_offs[i + 1] = p.plan.item_offs[i + 1];
        s_active[i] = p.plan.active[i];
        s_aoffs[i] = p.plan.aoffs[i];
        s_antok[i] = p.plan.antok[i];
    }
    if (tid == 0) s_item_offs[0] = 0;
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = tmem_slot;
    constexpr int RT = DUAL ? 64 : 128;                  // rows of one matrix an item covers
    const int nb = p.I / QK_K;
    const int n_mine = n_items > (int)blockIdx.x ? (n_items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    bool alive = true;
    const uint32_t bnr = (uint32_t)p.bnr, set_cols = NACC * bnr;   // a set of accumulators: the planes, then the mins
    constexpr uint32_t set_mask = TC_SETS - 1u;

    // Each warpgroup takes its share of the registers as it enters its branch; the branches do not meet before the end.
    if (warp < TC_CONV0) {
        // ------------------------------- drain ------------------------------------
        regs_inc<TC_REGS_DRAIN>();
        const int row = 32 * warp + lane;                // lane of tensor memory = row of the item
        const uint32_t lanes = tmem + ((uint32_t)(32 * warp) << 16);
        if (lane == 0 && n_mine > 0)                     // nothing was in the accumulators before
            for (int i = 0; i < TC_SETS; ++i) mbar_arrive(&in_full[i]);
        int sbg = 0, xph = 0;
        // the four warps meet (a barrier with a bounded wait, so that a warp that gave up leaves none of the others behind)
        auto meet = [&]() -> bool {
            __syncwarp();
            if (lane == 0) mbar_arrive(&x_bar);
            const bool ok = mbar_wait(&x_bar, xph);
            xph ^= 1;
            return ok;
        };
        for (int it = 0; it < n_mine && alive; ++it) {
            const int ir = it % TC_ITEMS;
            if (!mbar_wait_suspend(&item_full[ir], (it / TC_ITEMS) & 1)) {
                atomicExch(p.err, 11);
                break;
            }
            const int r0 = s_item[ir][1], np = s_item[ir][3];
            float f[BN], part[BN];                       // sums of the chains before, and of the chain at hand
#pragma unroll
            for (int j = 0; j < BN; ++j) f[j] = part[j] = 0.f;
#pragma unroll 1
            for (int b = 0; b < nb; ++b, ++sbg) {
                const uint32_t rs = (uint32_t)sbg % TC_RING, ph = ((uint32_t)sbg / TC_RING) & 1u;
                // its MMAs have finished; what came with its operands (scales in shared memory) is seen through the other barrier, long complete
                if (!mbar_wait_suspend(&done[rs], ph) || !mbar_wait(&in_full[rs], ph)) {
                    atomicExch(p.err, 11);
                    alive = false;
                    break;
                }
                tc_fence_after_sync();
                const uint32_t acc = lanes + ((uint32_t)sbg & set_mask) * set_cols;
                auto add = [&](auto width, const int c0) {
                    constexpr int W = decltype(width)::value;
                    uint32_t a[NACC][W];
#pragma unroll
                    for (int k = 0; k < NACC; ++k) tmem_ld_32xn(acc + k * bnr + c0, a[k]);
                    const uint32_t dd = s_meta[rs][row], dxa = smem_u32(&s_dx[rs][c0]);
                    const float dw = half_bits_to_float(dd) * (TYPE == IQ2_XXS ? 0.125f : 1.f), mw = half_bits_to_float(dd >> 16);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < W; j += 2) {
                        const uint4 dx = lds128(dxa + 8 * j);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const float x = __uint_as_float(h ? dx.z : dx.x);
                            const int c = (int)a[0][j + h];
                            float v;
                            if (TYPE == Q2_K) v = fmaf(dw, (float)c, -(mw * __uint_as_float(a[NACC - 1][j + h])));
                            else if (TYPE == Q3_K) v = dw * (float)((int)(h ? dx.w : dx.y) - c);
                            else v = dw * (float)(c + 128 * (int)a[NACC - 1][j + h]);
                            part[c0 + j + h] = fmaf(x, v, part[c0 + j + h]);
                        }
                    }
                };
                if (np <= 8) {
                    add(std::integral_constant<int, 8>(), 0);
                } else {
#pragma unroll
                    for (int c0 = 0; c0 < BN; c0 += 16) {
                        if (c0 >= np) break;
                        add(std::integral_constant<int, 16>(), c0);
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&in_full[(sbg + TC_SETS) % TC_RING]);
                if ((b & (TC_CHAIN - 1)) == TC_CHAIN - 1 || b == nb - 1) {
#pragma unroll
                    for (int c0 = 0; c0 < BN; c0 += 8) {
                        if (c0 >= np) break;
#pragma unroll
                        for (int j = c0; j < c0 + 8; ++j) { f[j] += part[j]; part[j] = 0.f; }
                    }
                }
            }
            if (!alive) break;
            // ---- the item is complete: activate, store ----
            // The columns' SwiGLU is a loop, not unrolled: the code runs once per item, and as a copy per column, each
            // skipped or not, it cost a miss of the instruction cache per copy, 10 us per item of 64 columns.
            const int row_out = r0 + (DUAL ? row & 63 : row);
            if (DUAL) {
                // gate rows are warps 0-1, up rows warps 2-3: through shared memory, then each thread takes every other column
#pragma unroll
                for (int j = 0; j < BN; j += 8) {
                    if (j >= np) break;
#pragma unroll
                    for (int k = j; k < j + 8; ++k) s_x[row * XP + k] = f[k];
                }
                if (!meet()) {
                    atomicExch(p.err, 21);
                    alive = false;
                }
                const int n = alive ? np : 0;
#pragma unroll 1
                for (int j = row >> 6; j < n; j += 2) {
                    const float g = s_x[(row & 63) * XP + j], u = s_x[(64 + (row & 63)) * XP + j];
                    if (row_out < p.O) {
                        count_bad(p.bad, g, u);
                        p.y[(size_t)s_pair[ir][j] * p.ldy + row_out] = swiglu_f(g, u, p.clamp, p.clamp_fused);
                    }
                }
                if (alive && !meet()) {
                    atomicExch(p.err, 21);
                    alive = false;
                }
            } else {
#pragma unroll
                for (int c0 = 0; c0 < BN; c0 += 8) {
                    if (c0 >= np) break;
#pragma unroll
                    for (int j = c0; j < c0 + 8; ++j)
                        if (j < np && row_out < p.O) p.y[(size_t)s_pair[ir][j] * p.ldy + row_out] = f[j];
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&item_empty[ir]);
        }
    } else if (warp < TC_TMA) {
        // ------------------------------- converters ------------------------------------
        // group g: half g % 2 of the super-blocks whose number has the parity g / 2
        regs_dec<TC_REGS_CONV>();
        const int cw = warp - TC_CONV0, q = cw & 3, n = (cw >> 2) & 1, par = cw >> 3;
        const int row = 32 * q + lane;
        const uint32_t lanes = tmem + ((uint32_t)(32 * q) << 16);
        // row r of a region of 64: G = 2^g_log2 sub-arrays, row G * sr + j in sub-array j at sr
        const int r = row & 63, gm = (1 << p.g_log2) - 1;
        const uint32_t row_at = raw_base + (uint32_t)(((row >> 6) * 64 + (r & gm) * (64 >> p.g_log2) + (r >> p.g_log2)) * p.pitch);
        const uint32_t row_off = (uint32_t)((r & gm) * p.rb);              // where the row starts in its group
        const bool uni = p.g_log2 == 0 || (TYPE == Q3_K || TYPE == IQ2_XXS ? p.g_log2 < 2 : false);
        const int cb = 1 << p.cb_log2, nch = (nb + cb - 1) >> p.cb_log2;
        int sbg0 = 0, rs = 0, rphase = 0;                    // super-blocks of the items before; the next chunk's raw stage
        // the super-block converted last: its stores may still be on their way
        int pending = -1;
        auto finish = [&]() {
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&in_full[pending % TC_RING]);
            pending = -1;
        };
        for (int it = 0; it < n_mine && alive; ++it, sbg0 += nb) {
            for (int c = 0; c < nch; ++c) {
                // every chunk is waited for and released, also one without a block for this group.  The stores before are handed over
                // while this half is loaded, or at once if its blocks are not there yet.
                if (!mbar_test_warp(&raw_full[rs], rphase)) {
                    if (pending >= 0) finish();
                    if (!mbar_wait_suspend(&raw_full[rs], rphase)) {
                        atomicExch(p.err, 12);
                        alive = false;
                        break;
                    }
                }
                const int r_now = rs, b0 = c << p.cb_log2, b = b0 + (((sbg0 + b0) ^ par) & 1), sbg = sbg0 + b;
                if (++rs == p.nraw) { rs = 0; rphase ^= 1; }
                if (b >= min(b0 + cb, nb)) {
                    if (lane == 0) mbar_arrive(&raw_empty[r_now]);
                    continue;
                }
                const uint32_t first = (uint32_t)(b0 * BB);
                TcHalf<TYPE> hf;
                hf.load(row_at + r_now * raw_bytes + ((row_off + first) & 15u) + ((uint32_t)(b * BB) - first), n, uni);
                if (pending >= 0) finish();
                uint32_t o[32];
                if constexpr (TYPE != IQ2_XXS) hf.conv(o);
                __syncwarp();
                if (lane == 0) mbar_arrive(&raw_empty[r_now]);
                if (sbg >= NA && !mbar_wait(&done[(sbg - NA) % TC_RING], ((sbg - NA) / TC_RING) & 1)) {
                    atomicExch(p.err, 13);
                    alive = false;
                    break;
                }
                tc_fence_after_sync();
                const uint32_t slot = lanes + A_COL + (uint32_t)(A_COLS * (sbg % NA));
                if constexpr (TYPE == IQ2_XXS) hf.store2(smem_u32(s_tab), slot + 32 * n);
                else tmem_st_32x32(slot + 32 * n, o);
                if constexpr (G::kMin) {
                    uint32_t mo[4];
                    hf.mins(mo);
                    tmem_st_32x4(slot + 64 * PL + 4 * n, mo);
                }
                if (n == 0) s_meta[sbg % TC_RING][row] = hf.d;
                pending = sbg;
            }
        }
        if (pending >= 0) finish();
    } else {
        regs_dec<TC_REGS_MISC>();
        if (warp == TC_TMA) {
        // ------------------------------- items and weight copies ------------------------------------
        const int nch = (nb + (1 << p.cb_log2) - 1) >> p.cb_log2, cbytes = BB << p.cb_log2, NG = 1 << p.g_log2;
        const int nrt = (p.O + RT - 1) / RT;
        const bool in_smem = n_active <= MMID_PLAN_SMEM;
        // item number it of this CTA: resolved and published, its pairs with it
        auto resolve = [&](int it, int &e, int &r0) -> bool {
            const int ir = it % TC_ITEMS;
            if (it >= TC_ITEMS && !mbar_wait_suspend(&item_empty[ir], ((it / TC_ITEMS) - 1) & 1)) return false;
            const int item = (int)blockIdx.x + it * (int)gridDim.x;
            // last a with item_offs[a] <= item: the lanes probe 32 points of the range at once
            int lo = 0, hi = n_active - 1;
            while (lo < hi) {
                const int step = (hi - lo + 31) >> 5, probe = min(hi, lo + (lane + 1) * step);
                const int v = in_smem ? s_item_offs[probe] : p.plan.item_offs[probe];
                const int k = __popc(__ballot_sync(0xffffffffu, v <= item));   // probes increase: a prefix of the lanes
                const int nlo = k == 0 ? lo : min(hi, lo + k * step);
                hi = max(nlo, k == 32 ? hi : min(hi, lo + (k + 1) * step) - 1);
                lo = nlo;
            }
            const int local = item - (in_smem ? s_item_offs[lo] : p.plan.item_offs[lo]);
            const int cnt = in_smem ? s_antok[lo] : p.plan.antok[lo], base = in_smem ? s_aoffs[lo] : p.plan.aoffs[lo];
            e = in_smem ? s_active[lo] : p.plan.active[lo];
            const int tc = local / nrt;
            r0 = (local - tc * nrt) * RT;
            // an expert's pairs are split evenly over its items: 65 pairs are 33 + 32, not 64 + 1
            const int n = (cnt + p.mt - 1) / p.mt, per = (cnt + n - 1) / n, np = min(per, cnt - tc * per);
            for (int i = lane; i < np; i += 32) s_pair[ir][i] = p.plan.slot[base + tc * per + i];
            if (lane == 0) *reinterpret_cast<int4 *>(s_item[ir]) = make_int4(e, r0, 0, np);
            __syncwarp();
            if (lane == 0) mbar_arrive(&item_full[ir]);
            return true;
        };
        int rs = 0, rphase = 1, e = 0, r0 = 0, e1 = 0, r1 = 0;   // the parity of the phase before the first counts as complete
        if (n_mine > 0) alive = resolve(0, e, r0);
        for (int it = 0; it < n_mine && alive; ++it) {
            for (int c = 0; c < nch; ++c) {
                if (!mbar_wait_suspend(&raw_empty[rs], rphase)) {
                    if (lane == 0) atomicExch(p.err, 14);
                    alive = false;
                    break;
                }
                if (lane == 0) mbar_arrive_expect_tx(&raw_full[rs], raw_bytes);
                __syncwarp();
                // copy j of a region brings, for each of its 64 / G row groups, the window that holds the chunk of row j of
                // the group, from the 16-byte boundary at or below its start; rows past the last arrive as zeros
                if (lane < 2 * NG) {
                    const int reg = lane >> p.g_log2, j = lane & (NG - 1);
                    tc_load_3d(raw_base + rs * raw_bytes + (uint32_t)((reg * 64 + j * (64 >> p.g_log2)) * p.pitch),
                               DUAL && reg ? &p.tm1 : &p.tm0, (j * p.rb + c * cbytes) & ~15, (r0 + (DUAL ? 0 : 64 * reg)) >> p.g_log2, e, &raw_full[rs]);
                }
                __syncwarp();
                if (++rs == p.nraw) { rs = 0; rphase ^= 1; }
                if (c == 0 && it + 1 < n_mine && !resolve(it + 1, e1, r1)) {
                    if (lane == 0) atomicExch(p.err, 19);
                    alive = false;
                    break;
                }
            }
            e = e1;
            r0 = r1;
        }
        } else if (warp == TC_MMA) {
        // ------------------------------- MMA issue ------------------------------------
        // values the same in all lanes and known as such (shuffles), one elected lane issues.  One barrier holds all that a
        // super-block's MMAs wait for: a wait that succeeds at once costs about 100 cycles.
        const uint32_t tbase = __shfl_sync(0xffffffffu, tmem, 0);
        const uint64_t desc0 = umma_desc_sw128(__shfl_sync(0xffffffffu, smem, 0));
        const uint64_t descm0 = umma_desc_sw32(__shfl_sync(0xffffffffu, bs_base, 0));
        const uint32_t atom = (uint32_t)p.bnr * 8u;      // 16-byte units between the two halves of an activation slot
        uint32_t sbg = 0;
        bool ready = false;                              // the next super-block's barrier, seen complete
        for (int it = 0; it < n_mine && alive; ++it) {
            const int ir = it % TC_ITEMS;
            if (!mbar_wait(&item_full[ir], (it / TC_ITEMS) & 1)) {
                if (lane == 0) atomicExch(p.err, 15);
                alive = false;
                break;
            }
            const int np = __shfl_sync(0xffffffffu, s_item[ir][3], 0);
            if (lane == 0) mbar_arrive(&item_empty[ir]);
            const int ncols = (np + 15) & ~15;
            const uint32_t idesc = umma_idesc_i8(128, ncols, TYPE == IQ2_XXS), idesc_m = umma_idesc_f16(128, ncols);
            for (int b = 0; b < nb; ++b, ++sbg) {
                const uint32_t set = sbg & set_mask, sb = sbg % TC_NB, nx = sbg + 1;
                if (!ready && !mbar_wait(&in_full[sbg % TC_RING], (sbg / TC_RING) & 1)) {
                    if (lane == 0) atomicExch(p.err, 16);
                    alive = false;
                    break;
                }
                ready = mbar_test_warp(&in_full[nx % TC_RING], (nx / TC_RING) & 1);
                tc_fence_after_sync();
                const uint32_t acc = tbase + set * set_cols, a0 = tbase + A_COL + A_COLS * (sbg % NA);
                const uint64_t b0 = desc0 + (uint64_t)(sb * (b_bytes >> 4));
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < 8; ++k)
#pragma unroll
                        for (int pl = 0; pl < PL; ++pl)
                            umma_i8_ta(acc + pl * bnr, a0 + 64 * pl + 8 * k, b0 + (k >> 2) * atom + 2 * (k & 3), idesc, k ? 1u : 0u);
                    if (G::kMin) umma_f16_ta(acc + PL * bnr, a0 + 64 * PL, descm0 + (uint64_t)(sb * bnr * 2u), idesc_m, 0u);
                    umma_commit(&done[sbg % TC_RING]);
                }
                __syncwarp();
            }
        }
        } else {
        // ------------------------------- activations ------------------------------------
        // Fill j brings super-block j of the CTA's run; the two warps take them in turn.  Sixteen lanes bring a row's 256 bytes, two its
        // fp16 group sums, one its d.  A warp has two fills on their way; it hands the older one over when the newer one is, or
        // while it has to wait for a slot.
        const int lw = warp - TC_LOAD0, c16 = lane & 15;
        const uint32_t src_off = (uint32_t)((c16 >> 2) * Q8_UNIT_STRIDE + 16 * (c16 & 3));
        const uint32_t dst_atom = (uint32_t)(c16 >> 3) * (uint32_t)p.bnr * 128u, cc = c16 & 7;
        uint32_t *const off = s_off[lw];
        int fill0 = 0;                                       // fills of the items before
        int pending = -1;
        auto complete = [&]() {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&in_full[pending % TC_RING]);
            pending = -1;
        };
        for (int it = 0; it < n_mine && alive; ++it, fill0 += nb) {
            const int ir = it % TC_ITEMS;
            if (!mbar_test_warp(&item_full[ir], (it / TC_ITEMS) & 1)) {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                if (pending >= 0) complete();
                if (!mbar_wait_suspend(&item_full[ir], (it / TC_ITEMS) & 1)) {
                    if (lane == 0) atomicExch(p.err, 20);
                    alive = false;
                    break;
                }
            }
            const int np = s_item[ir][3];
            __syncwarp();
#pragma unroll
            for (int i = 0; i < (BN + 31) / 32; ++i)
                if (32 * i + lane < np) off[32 * i + lane] = (uint32_t)(s_pair[ir][32 * i + lane] / p.xdiv) * (uint32_t)(p.q8_stride >> 4);
            __syncwarp();
            if (lane == 0) mbar_arrive(&item_empty[ir]);
            for (int b = (fill0 ^ lw) & 1; b < nb; b += 2) {
                const int fill = fill0 + b, slot = fill % TC_NB;
                if (fill >= TC_NB && !mbar_test_warp(&done[(fill - TC_NB) % TC_RING], ((fill - TC_NB) / TC_RING) & 1)) {
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                    if (pending >= 0) complete();
                    if (!mbar_wait_suspend(&done[(fill - TC_NB) % TC_RING], ((fill - TC_NB) / TC_RING) & 1)) {
                        if (lane == 0) atomicExch(p.err, 17);
                        alive = false;
                        break;
                    }
                }
                const uint8_t *const src = p.q8 + (size_t)b * Q8_BLOCK_STRIDE;
                const uint32_t dst = smem + slot * b_bytes + dst_atom;
#pragma unroll 4
                for (int i = 0; i < (np + 1) >> 1; ++i) {
                    const int rr = 2 * i + (lane >> 4);
                    if (rr < np)
                        cp_async_16(dst + (uint32_t)((rr >> 3) * 1024 + (rr & 7) * 128) + ((cc ^ (uint32_t)(rr & 7)) << 4), src + (size_t)off[rr] * 16 + src_off);
                }
                for (int i = 0; i < np; i += 16) {
                    const int rr = i + (lane >> 1), h = lane & 1;
                    if (rr < np) {
                        const uint8_t *const s2 = src + (size_t)off[rr] * 16;
                        if (G::kMin)
                            cp_async_16(bs_base + (uint32_t)((slot * p.bnr + rr) * 32 + 16 * (h ^ ((rr >> 2) & 1))), s2 + Q8_UNIT_STRIDE * h + 64);
                        if (h == 0) cp_async_8(smem_u32(&s_dx[fill % TC_RING][rr]), s2 + Q8_BLOCK_D);
                    }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                if (pending >= 0) {
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                    complete();
                }
                pending = fill;
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (pending >= 0) complete();
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

}  // namespace zmoe
