// dequant_f16.cuh -- half a super-block (128 consecutive weights of a quantised row) -> twice 64 fp16 values in 32 registers, in
// the order the prefill grouped GEMM stores them into tensor memory as one lane of its A operand.
//
// HalfBlock<TYPE> reads a copy of the super-block in shared memory (the grouped GEMM stages raw blocks there with
// the TMA engine).  Values follow the reference dequantisers (reference kernels/quant/kquant_matmul.cu:55-92,179-199,
// kernels/quant/iq2_matmul.cu:73-91): d*sc*q - dmin*m, d*(sc-32)*q3, d*(0.5+ls)*0.25*grid*sign, assembled directly in
// fp16: the integer part is exact, the block scale is rounded to fp16 once.
//
// What bounds the conversion: the integer pipe, which takes a warp instruction every other cycle (logic, shifts, selects, permutes),
// while the multiply-add pipes take one every cycle.  So a word of packed quants is shifted as little as possible: a field
// is masked where it sits in the mantissa of 1024 + field, and the multiply-add that takes 1024 off also divides by the field's place.
// Half a super-block per thread and not 64 weights, so that scales, high bits and the block's alignment are
// dealt with once for both steps; the scales are rounded as fp16 products (exact operands of at most 11 and 6 bits: the same single
// rounding as in f32).  Warp instructions per 64 weights, all / integer pipe, 64 weights at a time before -> now (with eight that store the
// result): Q2_K 237 / 126 -> 148 / 54, Q3_K 342 / 213 -> 211 / 107 (rows of different offsets 314 / 172 -> 198 / 95), Q4_K 198 / 91 -> 138 / 50,
// IQ2_XXS 280 / 165 -> 246 / 132.
//
// Order of k.  Register i of the 32 holds two weights; within every four consecutive k the pairs are (k, k+2) and
// (k+1, k+3), because masking a word of packed quants with 0x000F000F leaves bytes 0 and 2 in the two halves of a
// register: no byte permute is needed to assemble a pair.  A contraction does not care in which order k runs as long
// as both operands agree: the kernels that write the fp16 activations store each group of four in the order 0, 2, 1, 3
// (kpair_pack).
#pragma once

#include "quant_units.cuh"
#include "umma.cuh"

namespace zmoe {

// four consecutive activations -> the two fp16 pairs of the converters' k order
__device__ __forceinline__ uint2 kpair_pack(float v0, float v1, float v2, float v3) {
    return make_uint2(pack_f16x2(v0, v2), pack_f16x2(v1, v3));
}

// tables the converters read from shared memory
struct DequantTables {
    uint32_t grid;   // shared address of the IQ2_XXS selector table: 256 entries x IQ2_TABLE_COPIES copies x 16 bytes
};

// Entry e of the table: four byte-permute selectors, one per pair of elements (0, 2), (1, 3), (4, 6), (5, 7).  With
// i0, i1 the codes (0, 1, 2 for the magnitudes 8, 25, 43: their high nibbles) of the two elements, the
// selector's nibbles are (2 i0, 2 i0 + 1, 2 i1, 2 i1 + 1): the two bytes of each fp16 table entry.
// The table is kept in IQ2_TABLE_COPIES copies, entry e of copy c at index e * COPIES + c: lane l reads copy l % 8,
// so the eight lanes of a quarter-warp's 16-byte loads always fall into eight different groups of banks whatever
// entries the data asks for (one copy gave about three wavefronts per load from the data-dependent indices).
constexpr int IQ2_TABLE_COPIES = 8;
__device__ __forceinline__ void dequant_fill_tables(uint4 *grid_s) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        const uint64_t g = k_iq2xxs_grid[i];
        uint32_t w[4];
        for (int pp = 0; pp < 4; ++pp) {
            const int lo = 4 * (pp >> 1) + (pp & 1);      // elements lo and lo + 2
            const uint32_t i0 = (uint32_t)(g >> (8 * lo + 4)) & 3u, i1 = (uint32_t)(g >> (8 * lo + 20)) & 3u;
            w[pp] = 0x1010u + 0x22u * (i0 + 256u * i1);
        }
        for (int c = 0; c < IQ2_TABLE_COPIES; ++c) grid_s[i * IQ2_TABLE_COPIES + c] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }

// N words that start `off` bytes (0..15, even) into 16-byte chunks loaded with 128-bit loads: every lane reads another
// row, rows lie a multiple of 16 bytes apart, so 32-bit loads of one column meet four to a bank while a 128-bit load
// moves all four of its words through distinct banks.  The words are then picked with selects.
template <int N>
__device__ __forceinline__ void lds_window(uint32_t chunk, uint32_t off, uint32_t (&out)[N]) {
    constexpr int NC = (4 * N + 14 + 15) / 16;
    uint32_t c[4 * NC + 1];
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        const uint4 v = lds128(chunk + 16 * i);
        c[4 * i] = v.x; c[4 * i + 1] = v.y; c[4 * i + 2] = v.z; c[4 * i + 3] = v.w;
    }
    c[4 * NC] = 0;
    const bool two = off & 8, one = off & 4;
    constexpr int M = 4 * NC;
#pragma unroll
    for (int i = 0; i < M - 2; ++i) c[i] = two ? c[i + 2] : c[i];
#pragma unroll
    for (int i = 0; i < M - 3; ++i) c[i] = one ? c[i + 1] : c[i];
    const uint32_t sh = (off & 2) * 8;
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = __funnelshift_r(c[i], c[i + 1], sh);
}

// N words that start W words into 16-byte chunks, W known: 128-bit loads and no selects
template <int N, int W>
__device__ __forceinline__ void lds_words(uint32_t chunk, uint32_t (&out)[N]) {
    constexpr int NC = (N + W + 3) / 4;
    uint32_t c[4 * NC];
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        const uint4 v = lds128(chunk + 16 * i);
        c[4 * i] = v.x; c[4 * i + 1] = v.y; c[4 * i + 2] = v.z; c[4 * i + 3] = v.w;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = c[W + i];
}
template <int N, int W, bool HALVES>
__device__ __forceinline__ void lds_words_at(uint32_t at, uint32_t (&out)[N]) {
    if (HALVES && (at & 2u)) {
        uint32_t t[N + 1];
        lds_words<N + 1, W>(at & ~15u, t);
#pragma unroll
        for (int i = 0; i < N; ++i) out[i] = __funnelshift_r(t[i], t[i + 1], 16);
    } else {
        lds_words<N, W>(at & ~15u, out);
    }
}
// N words from an even address.  uniform: all lanes are as far from a 16-byte boundary; then the offset is a branch and no arithmetic.
// Otherwise rows of a group lie four words apart and 32-bit loads of one column fall into 32 banks.  HALVES: the address need not be
// a multiple of four.
template <int N, bool HALVES>
__device__ __forceinline__ void lds_span(uint32_t at, bool uniform, uint32_t (&out)[N]) {
    if (uniform) {
        const uint32_t w = (at >> 2) & 3u;
        if (w == 0) lds_words_at<N, 0, HALVES>(at, out);
        else if (w == 1) lds_words_at<N, 1, HALVES>(at, out);
        else if (w == 2) lds_words_at<N, 2, HALVES>(at, out);
        else lds_words_at<N, 3, HALVES>(at, out);
    } else if (HALVES && __any_sync(0xffffffffu, at & 2u)) {
        lds32xN_any<2, N>(at, out);
    } else {
        lds32xN_any<4, N>(at, out);
    }
}

// (a & b) | c in one instruction (written out: two constants among the operands came as two)
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
// (a & m) | (b & ~m), and (a & m) ^ b
__device__ __forceinline__ uint32_t bit_select(uint32_t m, uint32_t a, uint32_t b) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xCA;" : "=r"(r) : "r"(m), "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t and_xor(uint32_t a, uint32_t m, uint32_t b) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(r) : "r"(a), "r"(m), "r"(b));
    return r;
}

// fp16 pair (1024 + v * 2^S) -> v - B, exactly: times 2^-S, minus 1024 * 2^-S + B
template <int S, int B = 0>
__device__ __forceinline__ __half2 unmagic(uint32_t x) {
    if (S == 0) return __hsub2(bits_h2(x), __half2half2(__ushort_as_half(0x6400 + B)));
    constexpr float k = 1.f / (1 << S);
    return __hfma2(bits_h2(x), __float2half2_rn(k), __float2half2_rn(-1024.f * k - B));
}
template <int S, int B = 0>
__device__ __forceinline__ __half2 field(uint32_t x, uint32_t mask) { return unmagic<S, B>(and_or(x, mask, 0x64006400u)); }

// Half n of one row's super-block.  load takes what both steps need of it except, in Q4_K, the quants; step<S> gives the weights
// 128 n + 64 S and on, and calls `mid` halfway.  blk: shared address of the super-block's first byte (alignment as in the tensor: 2, 4 or 16
// bytes by type); uniform: the block's offset from a 16-byte boundary is the same for all rows.  Called by whole warps.
template <int TYPE> struct HalfBlock;

// IQ2_XXS: d @0, qs u16[32] @2.  The codebook holds only the magnitudes 8, 25 and 43, which index a three-entry fp16 table
// (the magnitudes times the sub-block scale) kept in a register pair; one byte permute per pair of
// elements assembles the values.  The shared-memory copy of the codebook holds, per entry, the four
// ready-made permute selectors instead of the magnitudes.
template <> struct HalfBlock<IQ2_XXS> {
    uint32_t aux[8];
    float d;
    uint32_t tcopy;
    __device__ __forceinline__ void load(uint32_t blk, int n, bool uniform, const DequantTables &tb) {
        lds_span<8, true>(blk + 2 + 32 * n, uniform, aux);
        d = half_bits_to_float(lds16(blk));
        tcopy = tb.grid + 16 * (threadIdx.x & (IQ2_TABLE_COPIES - 1));
    }
    template <int S, typename Mid> __device__ __forceinline__ void step(uint32_t (&o)[32], Mid mid) const {
#pragma unroll
        for (int ib = 0; ib < 2; ++ib) {
            if (ib == 1) mid();
            const uint32_t aux0 = aux[4 * S + 2 * ib], aux1 = aux[4 * S + 2 * ib + 1];
            const float db = __fmul_rn(__fmul_rn(d, 0.5f + (float)(aux1 >> 28)), 0.25f);
            const uint32_t t0 = h2_bits(__floats2half2_rn(db * 8.f, db * 25.f));   // entries 0, 1
            const uint32_t t1 = h2_bits(__floats2half2_rn(db * 43.f, 0.f));        // entry 2
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                const uint4 sel = lds128(tcopy + 16 * IQ2_TABLE_COPIES * __byte_perm(aux0, 0, 0x4440u | l));
                // Sign bits of the eight elements: the seven stored ones and their parity (even number of minus
                // signs per group of eight), bit 0 of the count.  One multiplication per pair (e, e + 2) moves bit e to bit 15
                // and bit e + 2 to bit 31: s * (2^(15 - e) + 2^(29 - e)) puts bit k of s at k + 15 - e and at k + 29 - e; the two
                // ranges are fourteen bits apart and s has ten (the count's upper bits are on top), so nothing carries, and
                // the mask keeps bits 15 and 31, which only bits e and e + 2 reach.
                const uint32_t s7 = (aux1 >> (7 * l)) & 127u;
                const uint32_t s8 = s7 + 128u * (uint32_t)__popc(s7);
                uint32_t *w = &o[16 * ib + 4 * l];
                w[0] = and_xor(s8 * 0x20008000u, 0x80008000u, __byte_perm(t0, t1, sel.x));
                w[1] = and_xor(s8 * 0x10004000u, 0x80008000u, __byte_perm(t0, t1, sel.y));
                w[2] = and_xor(s8 * 0x02000800u, 0x80008000u, __byte_perm(t0, t1, sel.z));
                w[3] = and_xor(s8 * 0x01000400u, 0x80008000u, __byte_perm(t0, t1, sel.w));
            }
        }
    }
};

// Q4_K: d @0, dmin @2, scales[12] @4, qs[128] @16.  nibble | 0x6400 is the fp16 number 1024 + q (1024 + 16 q for a high nibble left in
// place); taking 1024 off is exact, then one fused multiply-add per pair gives q * dl - ml.
template <> struct HalfBlock<Q4_K> {
    uint32_t at;
    __half2 dl[2], of[2];                          // scales and mins of sub-blocks (0, 2) and (1, 3) of the half
    __device__ __forceinline__ void load(uint32_t blk, int n, bool, const DequantTables &) {
        const uint4 h = lds128(blk);
        at = blk + 16 + 64 * n;
        // reference kernels/quant/kquant_matmul.cu:41-48
        uint32_t sc, mn;
        if (n == 0) {
            sc = h.y & 0x3F3F3F3Fu;
            mn = h.z & 0x3F3F3F3Fu;
        } else {
            sc = (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
            mn = ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
        }
        const __half2 d = __low2half2(bits_h2(h.x)), dmin = __hneg2(__high2half2(bits_h2(h.x)));
        dl[0] = __hmul2(d, field<0>(sc, 0x003F003Fu));
        dl[1] = __hmul2(d, field<0>(sc >> 8, 0x003F003Fu));
        of[0] = __hmul2(dmin, field<0>(mn, 0x003F003Fu));
        of[1] = __hmul2(dmin, field<0>(mn >> 8, 0x003F003Fu));
    }
    template <int S, typename Mid> __device__ __forceinline__ void step(uint32_t (&o)[32], Mid mid) const {
        const uint4 q0 = lds128(at + 32 * S), q1 = lds128(at + 32 * S + 16);
        const __half2 dl0 = S ? __high2half2(dl[0]) : __low2half2(dl[0]), dl1 = S ? __high2half2(dl[1]) : __low2half2(dl[1]);
        const __half2 of0 = S ? __high2half2(of[0]) : __low2half2(of[0]), of1 = S ? __high2half2(of[1]) : __low2half2(of[1]);
        const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const uint32_t x = w[m], y = w[m] >> 8;
            if (m == 4) mid();
            o[2 * m] = h2_bits(__hfma2(field<0>(x, 0x000F000Fu), dl0, of0));
            o[2 * m + 1] = h2_bits(__hfma2(field<0>(y, 0x000F000Fu), dl0, of0));
            o[16 + 2 * m] = h2_bits(__hfma2(field<4>(x, 0x00F000F0u), dl1, of1));
            o[16 + 2 * m + 1] = h2_bits(__hfma2(field<4>(y, 0x00F000F0u), dl1, of1));
        }
    }
};

// Q2_K: scales[16] @0, qs[64] @16, d @80, dmin @82; four two-bit planes of the 32 bytes that hold 128 weights
template <> struct HalfBlock<Q2_K> {
    uint32_t w[8], sc[2], dd;
    __device__ __forceinline__ void load(uint32_t blk, int n, bool uniform, const DequantTables &) {
        if (uniform) lds_span<8, false>(blk + 16 + 32 * n, true, w);
        else lds_window<8>((blk & ~15u) + 16 + 32 * n, blk & 12u, w);   // rows two words apart: see lds_window
        sc[0] = lds32(blk + 8 * n);
        sc[1] = lds32(blk + 8 * n + 4);
        dd = lds32(blk + 80);
    }
    template <int S, typename Mid> __device__ __forceinline__ void step(uint32_t (&o)[32], Mid mid) const {
        const __half2 d = __low2half2(bits_h2(dd)), dmin = __hneg2(__high2half2(bits_h2(dd)));
        // scales and mins of the groups of 16 numbers (0, 2) and (1, 3)
        const uint32_t s0 = sc[S], s1 = sc[S] >> 8;
        const __half2 dl02 = __hmul2(d, field<0>(s0, 0x000F000Fu)), dl13 = __hmul2(d, field<0>(s1, 0x000F000Fu));
        const __half2 of02 = __hmul2(dmin, field<4>(s0, 0x00F000F0u)), of13 = __hmul2(dmin, field<4>(s1, 0x00F000F0u));
        const __half2 dl[4] = {__low2half2(dl02), __low2half2(dl13), __high2half2(dl02), __high2half2(dl13)};
        const __half2 of[4] = {__low2half2(of02), __low2half2(of13), __high2half2(of02), __high2half2(of13)};
        constexpr uint32_t m0 = 0x00030003u << (4 * S), m1 = m0 << 2;
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const uint32_t x = w[m], y = w[m] >> 8;
            const int g = m >> 2;
            if (m == 4) mid();
            o[2 * m] = h2_bits(__hfma2(field<4 * S>(x, m0), dl[g], of[g]));
            o[2 * m + 1] = h2_bits(__hfma2(field<4 * S>(y, m0), dl[g], of[g]));
            o[16 + 2 * m] = h2_bits(__hfma2(field<4 * S + 2>(x, m1), dl[2 + g], of[2 + g]));
            o[16 + 2 * m + 1] = h2_bits(__hfma2(field<4 * S + 2>(y, m1), dl[2 + g], of[2 + g]));
        }
    }
};

// Q3_K: hmask[32] @0, qs[64] @32, scales[12] @96, d @108; four two-bit planes and the four matching planes of the high-bit mask
template <> struct HalfBlock<Q3_K> {
    uint32_t q[8], hm[8];                          // hm: the half's planes at bits 0..3 of every byte, the other's above (turned by 4 n)
    uint32_t s6[2];                                // the eight six-bit scales
    __half2 d;
    __device__ __forceinline__ void load(uint32_t blk, int n, bool uniform, const DequantTables &) {
        uint32_t t[3];
        lds_span<8, true>(blk, uniform, hm);
        lds_span<8, true>(blk + 32 + 32 * n, uniform, q);
        lds_span<3, true>(blk + 96, uniform, t);
        const uint32_t dd = lds16(blk + 108);
        d = __low2half2(bits_h2(dd));
#pragma unroll
        for (int i = 0; i < 8; ++i) hm[i] = n ? hm[i] >> 4 : hm[i];
        s6[0] = ((t[0] >> (4 * n)) & 0x0F0F0F0Fu) | (((t[2] >> (4 * n)) & 0x03030303u) << 4);
        s6[1] = ((t[1] >> (4 * n)) & 0x0F0F0F0Fu) | (((t[2] >> (4 * n + 2)) & 0x03030303u) << 4);
    }
    template <int S, typename Mid> __device__ __forceinline__ void step(uint32_t (&o)[32], Mid mid) const {
        const __half2 dl02 = __hmul2(d, field<0, 32>(s6[S], 0x003F003Fu)), dl13 = __hmul2(d, field<0, 32>(s6[S] >> 8, 0x003F003Fu));
        const __half2 dl[4] = {__low2half2(dl02), __low2half2(dl13), __high2half2(dl02), __high2half2(dl13)};
        // Fields of three bits where the quants sit: plane A at bit 4 S, plane B at bit 4 S + 2 of every byte, each with its high bit, which
        // takes the place of the next plane's first bit (of the next byte's, for the last plane: turned, so that none is lost).
        constexpr uint32_t qa = 0x03030303u << (4 * S), qb = qa << 2, fa = 0x00070007u << (4 * S), fb = fa << 2;
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            if (m == 4) mid();
            // high bits at 2 S and 2 S + 1: to 4 S + 2 and 4 S + 4
            const uint32_t ha = __funnelshift_l(hm[m], hm[m], 2 * S + 2), hb = __funnelshift_l(hm[m], hm[m], 2 * S + 3);
            const uint32_t a = bit_select(qa, q[m], ha), b = bit_select(qb, q[m], hb);
            const uint32_t a1 = __funnelshift_r(a, a, 8), b1 = __funnelshift_r(b, b, 8);
            const int g = m >> 2;
            o[2 * m] = h2_bits(__hmul2(field<4 * S, 4>(a, fa), dl[g]));
            o[2 * m + 1] = h2_bits(__hmul2(field<4 * S, 4>(a1, fa), dl[g]));
            o[16 + 2 * m] = h2_bits(__hmul2(field<4 * S + 2, 4>(b, fb), dl[2 + g]));
            o[16 + 2 * m + 1] = h2_bits(__hmul2(field<4 * S + 2, 4>(b1, fb), dl[2 + g]));
        }
    }
};

}  // namespace zmoe
