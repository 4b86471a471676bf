// gemm_sm100.cuh -- prefill-shaped grouped expert GEMM on the 5th-generation tensor
// cores: C[f, p] = sum_k W_e[f, k] * X[p, k] for the pairs p routed to expert e.
//
// Replaces, for calls with many tokens per expert, the GEMV-shaped per-expert loop of
// reference core/batched_dispatch_pipeline.cpp:1833-1921 and the dequantise-to-bf16 +
// cublasGemmEx escape hatch of reference backends/cuda/cuda_kernel_dispatcher.cpp:58-124.
//
// One persistent CTA per SM, warp-specialised.  A tile is 2 x 128 weight rows (DUAL: 128 gate
// rows and the same 128 up rows; otherwise rows m0..m0+127 and m0+128..m0+255 of one matrix)
// against up to 160 pairs; both halves multiply the same activation tile, which halves the
// activation traffic per flop.
//   warps 0, 3 issue tcgen05.mma (M = 128 weight rows, N = pairs, K = 16 per instruction, A from tensor memory, B from
//              shared memory), a half tile each; tcgen05.commit releases the operand slots.
//   warp 1     loader of the weights: copies the raw quantised super-blocks of the tile's 256 rows, one
//              super-block column (256 k) at a time, into a ring in shared memory with tiled copies on the TMA
//              engine (no multicast), completion on mbarriers.  Rows that are
//              not multiples of 16 bytes are addressed G rows at a time (G * row bytes is one): G
//              copies per 128 rows, one per position of a row inside its group.
//   warp 2     loader of the activations: one tiled copy per 64 k of the rows gathered into expert order, into a
//              ring of its own.
//   warps 4-19 converters, two groups of eight: a thread reads 128 consecutive weights of one row from shared memory,
//              converts 64 at a time to fp16 in 32 registers and stores them as its lane of the A operand in tensor memory.
//              The groups take alternate k-steps (each has a half of the super-block), so that one group's loads and conversion
//              overlap the other's waits.  A group converts before it waits for its operand slot and loads its next half before it needs it.
//   warps 20-23 drain the accumulators of a finished tile (tcgen05.ld, SwiGLU in DUAL mode, f32 stores).
//
// What bounds it.  A from tensor memory: with both operands in shared memory the fp16 weights cost a store and a read there
// (16 KB each per half tile and k-step), and raw blocks, activations, stores and operand reads together needed more
// shared-memory cycles than the MMAs take tensor cycles.  Tensor memory (512 columns) holds two accumulators of 160 columns
// and three operand slots of 2 x 32, hence 160 pairs per tile: the way round from a slot's release to its next use
// (commit, wait, tcgen05.st, wait, issue) takes longer than the MMAs of one other slot.  Tiles of at most
// 80 pairs use half of the accumulator columns and alternate between two buffers, so that the
// drain of one overlaps the MMAs of the next.  Below about 100 pairs the converters' instruction issue is the limit (every
// weight is converted once per pair block): 64 % of the issue slots at 44 pairs, the integer pipe half busy.
// Measured on one B200, layers of 128 experts, us per layer with all its launches, the same layer and input called over and over, this form against
// one where sixteen warps converted 64 weights at a time and drained as well and one warp issued all MMAs: 4096 / 1536, Q2_K gate and up, Q3_K down, 512
// tokens 760 -> 548, 700 785 -> 576, 1024 831 -> 624; IQ2_XXS 700 tokens 836 -> 637; Q3_K 700 928 -> 671; Q4_K 2048 / 768 512 tokens 247 -> 189.
// With layers and inputs that change from call to call: 700 tokens 785 -> 616; 4096 tokens of IQ2_XXS, skewed load, 2351 -> 2058; 8192 tokens of 7168 / 2048, 256
// experts, Q4_K, with a shared expert 10 250 -> 8 820.
// Tiles of more than 80 pairs wait for the drain of the one before: its instructions per column count (35 -> about 20 by a loop without clamps,
// 128-bit loads of the columns' scales and pairs and no predicates on full chunks: 4096 tokens 1908 -> 1734 and, Q4_K 2048 / 768, 775 -> 645).
// Eight drain warps instead of four took 1718 and 643 there, but 617 instead of 587 at 700 tokens; a drain that loads the next columns
// ahead was slower (more moves), waits that sleep instead of polling made no difference.
// Activations arrive already rounded through Q8_K (value = d * q) as fp16, each row divided by a
// power of two that brings its largest value near 2^13 (undone exactly in the epilogue), so the
// result follows the reference CPU path's activation quantisation and cannot overflow fp16;
// weights are fp16 too (dequant_f16.cuh): exact integer part, block scale and min each rounded once, then one fp16 multiplication or multiply-add.
// A weight is off by at most 2^-11 of itself for that and 2^-11 of the scaled part and of the min (IQ2_XXS: one rounding of a scaled magnitude).
// Every wait is bounded; on expiry the CTA raises the error flag and unwinds, and the
// tensor memory is always released.
#pragma once

#include <cuda.h>

#include "dequant_f16.cuh"
#include "mmid.cuh"

namespace zmoe {

constexpr int GEMM_BM = 128;        // weight rows per half tile
constexpr int GEMM_BN = 160;        // pairs per tile (tensor-memory columns per accumulator)
constexpr int GEMM_BK = 64;         // k per step: one 128-byte swizzle row of fp16 activations, 32 columns of fp16 weights
constexpr int GEMM_NB = 4;          // activation slots
constexpr int GEMM_NRAW = 3;        // raw super-block slots
constexpr int GEMM_CWARPS = 16;     // converter warps: two groups of eight
constexpr int GEMM_CW0 = 4;          // first of them, a multiple of four
constexpr int GEMM_DW0 = GEMM_CW0 + GEMM_CWARPS;   // first of the four drain warps
constexpr int GEMM_THREADS = 32 * (GEMM_DW0 + 4);
constexpr int GEMM_NA = 3;          // weight slots in tensor memory, 2 x 32 columns each
constexpr int GEMM_A_COL = 2 * GEMM_BN;   // tensor-memory column of the first of them
constexpr int GEMM_NBOX = GEMM_BN / 32;   // activation boxes of 32, 64, .. 160 rows
constexpr int GEMM_MAX_ACTIVE = 512;
// registers per thread: of the launch, and of the warpgroups' roles, which add up to six times the launch's
constexpr int GEMM_REGS = 80, GEMM_REGS_CONV = 88, GEMM_REGS_DRAIN = 80, GEMM_REGS_MISC = 48;
static_assert(4 * GEMM_REGS_CONV + GEMM_REGS_DRAIN + GEMM_REGS_MISC == 6 * GEMM_REGS, "registers");

// bytes between the raw copies of consecutive rows in shared memory: room for one super-block plus its
// offset from the 16-byte boundary the copy starts on, and a multiple of 16 that is 16 or 48 modulo 128
// so that the converters' loads (one row per lane pair) spread over the banks
template <int TYPE> struct RawGeom;
template <> struct RawGeom<IQ2_XXS> { static constexpr int kPitch = 80; };    // 66 + 14
template <> struct RawGeom<Q2_K> { static constexpr int kPitch = 112; };      // 84 + 12
template <> struct RawGeom<Q3_K> { static constexpr int kPitch = 144; };      // 110 + 14
template <> struct RawGeom<Q4_K> { static constexpr int kPitch = 144; };      // 144 + 0
__host__ __device__ constexpr int gemm_raw_pitch(int type) {
    return type == IQ2_XXS ? 80 : type == Q2_K ? 112 : 144;
}

struct GemmParams {
    const uint8_t *w0, *w1;      // quantised weights (w1: up, DUAL only)
    size_t stride0, stride1;     // bytes between experts
    int I, O;                    // k extent, weight rows per expert (multiple of 128)
    int rb;                      // bytes per weight row
    int g_log2;                  // log2 of G, the rows per group whose bytes are a multiple of 16 (1, 2, 4 or 8 rows)
    const float *xscale;         // per SORTED activation row: the power of two the row was divided by
    float *y;                    // output [pair][ldy]
    int ldy;
    const int *hdr, *active, *aoffs, *antok, *slot;   // plan (see router.cuh)
    float clamp;
    int clamp_fused;
    int *err;
    int *bad;                    // DUAL: [2] counters of NaN / Inf gate or up values, or null
    unsigned long long *stats;   // cycle counters of CTA 0's roles (builds with ZMOE_GEMM_STATS only), or null
};

// Cycle accounting of one CTA's roles, compiled in with -DZMOE_GEMM_STATS (python -m zeromoe_b200.build with
// ZMOE_GEMM_STATS=1 in the environment): one thread per role of CTA 0 adds up clock64() differences around
// its waits and its work and stores the sums when the kernel ends.  Slots: 0 k-steps, 1 converter
// wait for raw blocks, 2 load + convert, 3 drain, 4 wait for an operand slot, 5 store + arrive,
// 6 MMA wait for operands, 7 drain wait for the accumulators, 8 MMA wait for the accumulators, 9 tiles,
// 10 MMA issue.
#ifdef ZMOE_GEMM_STATS
#define GSTAT_DECL unsigned long long gs_t0 = 0, gs_acc[5] = {0, 0, 0, 0, 0}; const bool gs_on = blockIdx.x == 0 && p.stats != nullptr
#define GSTAT_BEGIN() do { if (gs_on) gs_t0 = clock64(); } while (0)
#define GSTAT_END(i) do { if (gs_on) { const unsigned long long gs_t1 = clock64(); gs_acc[i] += gs_t1 - gs_t0; gs_t0 = gs_t1; } } while (0)
#define GSTAT_STORE(i, slot) do { if (gs_on) p.stats[slot] += gs_acc[i]; } while (0)
#define GSTAT_COUNT(n, slot) do { if (gs_on) p.stats[slot] += (unsigned long long)(n); } while (0)
#else
#define GSTAT_DECL do { } while (0)
#define GSTAT_BEGIN() do { } while (0)
#define GSTAT_END(i) do { } while (0)
#define GSTAT_STORE(i, slot) do { } while (0)
#define GSTAT_COUNT(n, slot) do { } while (0)
#endif

// Activation tile maps with boxes of 32, 64, .. 160 rows (a tile loads the smallest box that covers
// its pairs, so an expert with few pairs does not pull 160 rows through L2 for every k-step) and the
// byte maps [E][O / G][G * rb] of the weight tensors with a box of 128 / G row groups x one raw row pitch.
struct GemmMaps {
    alignas(64) CUtensorMap box[GEMM_NBOX];
    alignas(64) CUtensorMap wmap[2];
};

// 3-D tiled copy (no multicast): box of the map at (x, row, expert); x must be a multiple of 16 bytes
__device__ __forceinline__ void tma_load_3d(uint32_t dst_smem, const void *tmap, int x, int row, int expert, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst_smem), "l"(tmap), "r"(x), "r"(row), "r"(expert), "r"(smem_u32(bar))
        : "memory");
}

template <int TYPE, bool DUAL>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_sm100_kernel(const GemmParams p, const __grid_constant__ GemmMaps maps) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // K-step j of the CTA's run (counted through its tiles) uses entry j % GEMM_NB of two rings: in_full, all that its MMAs wait for (the
    // weights from eight converter warps, the activations), and done, its MMAs (of both issuers) have finished: its operand slots can be
    // refilled.  No waiter can be a whole ring behind: each arrives on the in_full of a later k-step first.
    // raw_*: raw super-block slots; acc_*: accumulator buffers, by tile parity
    __shared__ __align__(8) uint64_t in_full[GEMM_NB], done[GEMM_NB], raw_full[GEMM_NRAW], raw_empty[GEMM_NRAW], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_tile_offs[GEMM_MAX_ACTIVE + 1], s_active[GEMM_MAX_ACTIVE], s_aoffs[GEMM_MAX_ACTIVE], s_antok[GEMM_MAX_ACTIVE];
    __shared__ __align__(16) int2 s_col[4][GEMM_BN];                       // per drain warp: scale (as bits) and pair of a tile's columns
    __shared__ __align__(16) uint4 grid_s[TYPE == IQ2_XXS ? 256 * IQ2_TABLE_COPIES : 1];

    // 1024-byte alignment of the activation tiles (required by the 128-byte swizzle)
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    constexpr int BB = QTraits<TYPE>::kBytes;
    constexpr int PITCH = RawGeom<TYPE>::kPitch;
    constexpr int B_BYTES = GEMM_BN * GEMM_BK * 2;           // 20 KB
    constexpr int RAW_HALF = GEMM_BM * PITCH;                // raw blocks of one half tile
    constexpr int RAW_SLOT = 2 * RAW_HALF;
    constexpr uint32_t TMEM_COLS = 512;
    uint8_t *raw_base = smem + GEMM_NB * B_BYTES;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(&acc_full[s], 2);                 // a commit of each issuer
            mbar_init(&acc_empty[s], 4);
        }
        for (int s = 0; s < GEMM_NB; ++s) {
            mbar_init(&in_full[s], GEMM_CWARPS / 2 + 1);   // one arrival per warp of the group, the loader's expect_tx arrival
            mbar_init(&done[s], 2);
        }
        for (int s = 0; s < GEMM_NRAW; ++s) {
            mbar_init(&raw_full[s], 1);
            mbar_init(&raw_empty[s], GEMM_CWARPS);
        }
        mbar_init_fence();
    }
    if (warp == 0) tmem_alloc(&tmem_slot, TMEM_COLS);
    if (TYPE == IQ2_XXS) dequant_fill_tables(grid_s);
    const DequantTables tb{smem_u32(grid_s)};

    pdl_wait_prior_grid();
    pdl_launch_dependents();

    // tiles: for each active expert, row blocks x ceil(pairs / 160) pair blocks
    const int n_active = min(p.hdr[0], GEMM_MAX_ACTIVE);
    const int mstep = DUAL ? GEMM_BM : 2 * GEMM_BM;          // rows of one matrix a tile covers
    const int mblocks = (p.O + mstep - 1) / mstep;
    for (int i = tid; i < n_active; i += GEMM_THREADS) {
        s_active[i] = p.active[i];
        s_aoffs[i] = p.aoffs[i];
        s_antok[i] = p.antok[i];
    }
    if (warp == 0) {
        // prefix sums of the tiles per active expert, 32 experts at a time
        int run = 0;
        if (lane == 0) s_tile_offs[0] = 0;
        for (int a0 = 0; a0 < n_active; a0 += 32) {
            const int a = a0 + lane;
            int v = a < n_active ? mblocks * ((p.antok[a] + GEMM_BN - 1) / GEMM_BN) : 0;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int o = __shfl_up_sync(0xffffffffu, v, off);
                if (lane >= off) v += o;
            }
            if (a < n_active) s_tile_offs[a + 1] = run + v;
            run += __shfl_sync(0xffffffffu, v, 31);
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_slot;
    const int n_tiles = s_tile_offs[n_active];
    const int ksteps = p.I / GEMM_BK;                        // a multiple of four
    const int nblk = p.I / QK_K;
    bool alive = true;

    // which expert, rows and pairs a tile has; called by whole warps
    auto tile_info = [&](int tile, int &e, int &m0, int &p0, int &np) {
        // last a with s_tile_offs[a] <= tile: the lanes probe 32 points of the range at once
        int lo = 0, hi = n_active - 1;
        while (lo < hi) {
            const int step = (hi - lo + 31) >> 5, probe = min(hi, lo + (lane + 1) * step);
            const int k = __popc(__ballot_sync(0xffffffffu, s_tile_offs[probe] <= tile));   // probes increase: a prefix of the lanes
            const int nlo = k == 0 ? lo : min(hi, lo + k * step);
            hi = max(nlo, k == 32 ? hi : min(hi, lo + (k + 1) * step) - 1);
            lo = nlo;
        }
        const int local = tile - s_tile_offs[lo];
        e = s_active[lo];
        // pair block outermost: the row blocks of one pair block run back to back and reuse
        // the same activation rows from L2
        const int nb = local / mblocks;
        m0 = (local % mblocks) * mstep;
        // an expert's pairs are split evenly over its pair blocks (180 pairs: 96 + 84, not 160 + 20)
        const int cnt = s_antok[lo], npb = (cnt + GEMM_BN - 1) / GEMM_BN;
        const int bsz = ((cnt + npb - 1) / npb + 15) & ~15;
        p0 = s_aoffs[lo] + nb * bsz;
        np = max(0, min(bsz, cnt - nb * bsz));
    };
    // the second half of a tile exists unless the matrix ends after the first (rows a multiple of 128, not 256)
    auto has_half1 = [&](int m0) -> bool { return DUAL || m0 + GEMM_BM < p.O; };
    // accumulators of tile number nt of this CTA: column of the first one and distance to the second
    auto acc_col = [&](int nt, int np) -> uint32_t { return np <= GEMM_BN / 2 ? (uint32_t)((nt & 1) * GEMM_BN) : 0u; };
    auto acc_stride = [&](int np) -> uint32_t { return np <= GEMM_BN / 2 ? GEMM_BN / 2 : GEMM_BN; };

    if (warp >= GEMM_CW0 && warp < GEMM_DW0) {
        // ------------------------------- converters ------------------------------------
        regs_inc<GEMM_REGS_CONV>();
        // thread -> (group, half tile, row); a warp may only touch the quarter warp % 4 of the tensor-memory lanes
        const int cw = warp - GEMM_CW0;
        const int q = cw & 3, which = (cw >> 2) & 1, grp = cw >> 3;
        const int r = 32 * q + lane;
        const uint32_t lanes = tmem_base + ((uint32_t)(32 * q) << 16);
        const uint32_t a_slot = lanes + GEMM_A_COL + 32 * which;
        // row r = G * sr + j sits in sub-array j (the copy of position j of every group) at sr
        const int G = 1 << p.g_log2, rj = r & (G - 1), rsr = r >> p.g_log2;
        const uint32_t row_at = smem_u32(raw_base) + which * RAW_HALF + (rj * (GEMM_BM >> p.g_log2) + rsr) * PITCH;
        uint32_t col = 0;                     // super-block columns so far: column col holds k-steps 4 col to 4 col + 3
        uint32_t rs = 0, rph = 0;             // its raw slot, and that one's phase
        uint32_t slot = grp;                  // operand slot of this group's next k-step
        GSTAT_DECL;
        HalfBlock<TYPE> hb;
        // the half of column col, super-block b of its tile (rows of a half tile that does not exist: what lies there, never stored)
        auto load = [&](int b) -> bool {
            if (!mbar_wait(&raw_full[rs], rph)) {
                atomicExch(p.err, 7);
                return false;
            }
            hb.load(row_at + rs * RAW_SLOT + ((uint32_t)(rj * p.rb + b * BB) & 15u), grp, p.g_log2 == 0, tb);
            return true;
        };
        // The k-step stored last, whose stores may still be on their way.  It is handed over at once, since the MMAs of all k-steps come
        // one after the other and a late one holds up the three operand slots, or halfway through the next one's conversion (us per
        // layer, at once / halfway: Q2_K and Q3_K 700 tokens 569 / 582, Q4_K 2048 / 768 512 tokens 196 / 201, 7168 / 2048 8192 tokens 8183 / 8465;
        // IQ2_XXS, whose conversion is the longest, 512 tokens 632 / 622).
        constexpr bool LATE = TYPE == IQ2_XXS;
        int pending = -1;
        auto finish = [&]() {
            if (pending < 0) return;
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&in_full[pending]);
            pending = -1;
        };
        const auto midway = [&] { if (LATE) finish(); };
        if ((int)blockIdx.x < n_tiles) alive = load(0);
        for (int tile = blockIdx.x; alive && tile < n_tiles; tile += gridDim.x) {
            int e, m0, p0, np;
            tile_info(tile, e, m0, p0, np);
            const bool worker = which == 0 || has_half1(m0);
            // k-step 4 col + e into its operand slot, which was last read by the k-step three before: the next entry of the ring, of this
            // column for the last step and of the one before for the others (before the first column: a phase that counts as complete).
            uint32_t a[32];
            auto put = [&](const uint32_t e) -> bool {
                const uint32_t before = (e + 1) % GEMM_NB;
                if (!mbar_wait(&done[before], (col + (before == 0 ? 0 : 1)) & 1)) {
                    atomicExch(p.err, 3);
                    return false;
                }
                GSTAT_END(3);
                tc_fence_after_sync();
                if (worker) tmem_st_32x32(a_slot + 64 * slot, a);
                pending = (int)e;
                slot = slot == 0 ? GEMM_NA - 1 : slot - 1;        // two steps on
                if (!LATE) finish();
                GSTAT_END(4);
                return true;
            };
            // the groups take alternate k-steps: 4 col + grp and 4 col + 2 + grp are the two of this group's half
            for (int b = 0; b < nblk; ++b) {
                GSTAT_BEGIN();
                if (worker) hb.template step<0>(a, midway);
                else midway();
                GSTAT_END(1);
                if (!put(grp)) {
                    alive = false;
                    break;
                }
                if (worker) hb.template step<1>(a, midway);
                else midway();
                __syncwarp();
                if (lane == 0) mbar_arrive(&raw_empty[rs]);       // this warp is done with the raw slot
                GSTAT_END(1);
                if (!put(2 + grp)) {
                    alive = false;
                    break;
                }
                ++col;
                if (++rs == GEMM_NRAW) { rs = 0; rph ^= 1; }
                if ((b + 1 < nblk || tile + (int)gridDim.x < n_tiles) && !load(b + 1 < nblk ? b + 1 : 0)) {
                    alive = false;
                    break;
                }
                GSTAT_END(0);
            }
        }
        finish();
#ifdef ZMOE_GEMM_STATS
        if (cw == 1 && lane == 0) {
            GSTAT_COUNT(4 * col, 0);
            GSTAT_STORE(0, 1); GSTAT_STORE(1, 2); GSTAT_STORE(3, 4); GSTAT_STORE(4, 5);
        }
#endif
    } else if (warp >= GEMM_DW0) {
        // ------------------------------- drain ------------------------------------
        // Warp w reads its quarter of the lanes (rows) of a finished tile's accumulators, eight columns (pairs) at a time.  The
        // loop over the columns stays rolled: the code runs once per tile and would otherwise be fetched anew each time.
        const int q = warp & 3;
        const uint32_t lanes = tmem_base + ((uint32_t)(32 * q) << 16);
        const bool plain = p.clamp <= 0.f;                       // then both forms of the activation are the same
        int nt = 0;
        GSTAT_DECL;
        for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++nt) {
            int e, m0, p0, np;
            tile_info(tile, e, m0, p0, np);
            const bool two = has_half1(m0);
            __syncwarp();
            for (int c = lane; c < ((np + 7) & ~7); c += 32)
                s_col[q][c] = c < np ? make_int2(__float_as_int(p.xscale[p0 + c]), p.slot[p0 + c]) : make_int2(0, 0);
            __syncwarp();
            GSTAT_BEGIN();
            if (!mbar_wait_suspend(&acc_full[nt & 1], (nt >> 1) & 1)) {
                atomicExch(p.err, 6);
                break;
            }
            GSTAT_END(0);
            tc_fence_after_sync();
            const uint32_t acc0 = lanes + acc_col(nt, np), acc1 = acc0 + acc_stride(np);
            float *const yf = p.y + m0 + 32 * q + lane;          // this thread's weight row (first half)
#pragma unroll 1
            for (int c0 = 0; c0 < np; c0 += 8) {
                uint32_t g[8], u[8];
                tmem_ld_32x8(acc0 + c0, g);
                if (two) tmem_ld_32x8(acc1 + c0, u);
                int4 m[4];                                       // scale and pair of columns 2 i and 2 i + 1
#pragma unroll
                for (int i = 0; i < 4; ++i) m[i] = *reinterpret_cast<const int4 *>(&s_col[q][c0 + 2 * i]);
                tmem_ld_wait();
                // x * 0 is 0 for a finite x and NaN otherwise: the sum flags a value that is not finite, as every result of a gate or up
                // value that is not finite is
                float probe = 0.f;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float sc = __int_as_float(j & 1 ? m[j >> 1].z : m[j >> 1].x);
                    const float gv = __uint_as_float(g[j]) * sc;
                    if (DUAL) {
                        const float uv = __uint_as_float(u[j]) * sc;
                        float v;
                        if (plain) {
                            v = swiglu_fast(gv, uv, 0.f, 0);
                            probe = fmaf(v, 0.f, probe);
                        } else {
                            probe = fmaf(gv, 0.f, fmaf(uv, 0.f, probe));
                            v = swiglu_fast(gv, uv, p.clamp, p.clamp_fused);
                        }
                        g[j] = __float_as_uint(v);
                    } else {
                        g[j] = __float_as_uint(gv);
                        if (two) u[j] = __float_as_uint(__uint_as_float(u[j]) * sc);
                    }
                }
                auto store = [&](int j) {
                    float *row = yf + (size_t)(uint32_t)(j & 1 ? m[j >> 1].w : m[j >> 1].y) * (uint32_t)p.ldy;
                    row[0] = __uint_as_float(g[j]);
                    if (!DUAL && two) row[GEMM_BM] = __uint_as_float(u[j]);
                };
                if (c0 + 8 <= np) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) store(j);
                } else {
#pragma unroll
                    for (int j = 0; j < 7; ++j)
                        if (c0 + j < np) store(j);
                }
                // warp-uniform decision: the loads below are warp-collective
                if (DUAL && p.bad && __any_sync(0xffffffffu, probe != probe)) {
                    // rare: recount this chunk's non-finite inputs exactly
#pragma unroll 1
                    for (int j = 0; j < 8; ++j) {
                        uint32_t gj, uj;
                        tmem_ld_1(acc0 + c0 + j, gj);
                        tmem_ld_1(acc1 + c0 + j, uj);
                        tmem_ld_wait();
                        const float sc = __int_as_float(s_col[q][c0 + j].x);
                        if (c0 + j < np) count_bad(p.bad, __uint_as_float(gj) * sc, __uint_as_float(uj) * sc);
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[nt & 1]);
            GSTAT_END(2);
        }
#ifdef ZMOE_GEMM_STATS
        if (q == 1 && lane == 0) { GSTAT_STORE(0, 7); GSTAT_STORE(2, 3); }
#endif
    } else {
        regs_dec<GEMM_REGS_MISC>();
        if (warp == 0 || warp == 3) {
        // ------------------------------- MMA issuers ------------------------------------
        // One warp per half tile: at the few instructions a lone warp gets through between sixteen converter warps, the eight MMAs of a
        // k-step, their addresses and two commits took one warp 474 cycles where the tensor core takes 195 (48 pairs).
        // The whole warp runs this loop on values that are the same in all lanes and known to the compiler as such
        // (shuffles from lane 0), and one elected lane issues: the operands then live in uniform registers.  With a
        // branch on the lane number every operand of every MMA was moved there one by one.
        int nt = 0;
        uint32_t it = 0, s = 0;                                     // k-steps so far; operand slot of the next
        const uint32_t tbase = __shfl_sync(0xffffffffu, tmem_base, 0);
        const uint64_t desc_b0 = umma_desc_sw128(__shfl_sync(0xffffffffu, smem_u32(smem), 0));   // a k-step of 16 advances the start address by 32 bytes
        const uint32_t half = __shfl_sync(0xffffffffu, warp == 0 ? 0u : 1u, 0);
        bool ready = false;                                         // the next k-step's operands, seen complete
        bool small_before = true;                                   // the tile before used one of the two small buffers
        GSTAT_DECL;
        for (int tile = blockIdx.x; tile < n_tiles && alive; tile += gridDim.x, ++nt) {
            int e, m0, p0, np;
            tile_info(tile, e, m0, p0, np);
            np = __shfl_sync(0xffffffffu, np, 0);
            m0 = __shfl_sync(0xffffffffu, m0, 0);
            const int ncols = (np + 15) & ~15;
            const uint32_t idesc = umma_idesc_f16(GEMM_BM, ncols);
            const bool mine = half == 0 || has_half1(m0), small = np <= GEMM_BN / 2;
            const uint32_t d = tbase + acc_col(nt, np) + half * acc_stride(np);
            GSTAT_BEGIN();
            // what this tile's accumulators overwrite must have been drained: always the tile two before, and the
            // one before unless both fit the two small buffers
            if ((nt >= 2 && !mbar_wait_suspend(&acc_empty[nt & 1], ((nt >> 1) - 1) & 1)) ||
                (nt >= 1 && !(small && small_before) && !mbar_wait_suspend(&acc_empty[(nt - 1) & 1], ((nt - 1) >> 1) & 1))) {
                if (lane == 0) atomicExch(p.err, 4);
                alive = false;
                break;
            }
            small_before = small;
            GSTAT_END(2);
            uint32_t acc = 0;
            for (int left = ksteps; left > 0; --left, ++it) {
                const uint32_t sb = it % GEMM_NB;
                GSTAT_BEGIN();
                if (!ready && !mbar_wait(&in_full[sb], (it / GEMM_NB) & 1)) {
                    if (lane == 0) atomicExch(p.err, 5);
                    alive = false;
                    break;
                }
                GSTAT_END(0);
                // Issuing blocks until the tensor core has taken the MMAs, and a wait that succeeds at once still costs
                // about 100 cycles: the next step's operands are looked at before this step's MMAs go out, so that the
                // answer is there when they have.
                const uint32_t nx = it + 1;
                ready = mbar_test_wait(&in_full[nx % GEMM_NB], (nx / GEMM_NB) & 1);
                tc_fence_after_sync();
                if (elect_one()) {
                    if (mine) {
                        const uint32_t a0 = tbase + GEMM_A_COL + 64 * s + 32 * half;
                        const uint64_t b0 = desc_b0 + (uint64_t)(sb * (B_BYTES >> 4));
#pragma unroll
                        for (int k4 = 0; k4 < GEMM_BK / 16; ++k4) umma_f16_ta(d, a0 + 8 * k4, b0 + 2 * k4, idesc, k4 ? 1u : acc);
                    }
                    umma_commit(&done[sb]);                         // both operands are free once these MMAs have read them
                    if (left == 1) umma_commit(&acc_full[nt & 1]);  // accumulators complete
                }
                s = s == GEMM_NA - 1 ? 0 : s + 1;
                __syncwarp();
                acc = 1;
                GSTAT_END(3);
            }
        }
#ifdef ZMOE_GEMM_STATS
        if (warp == 0 && lane == 0) { GSTAT_STORE(0, 6); GSTAT_STORE(2, 8); GSTAT_COUNT(nt, 9); GSTAT_STORE(3, 10); }
#endif
    } else if (warp == 1) {
        // ------------------------------- weight loader ------------------------------------
        int rc = 0;
        for (int tile = blockIdx.x; tile < n_tiles && alive; tile += gridDim.x) {
            int e, m0, p0, np;
            tile_info(tile, e, m0, p0, np);
            const bool two = has_half1(m0);
            for (int b = 0; b < nblk; ++b, ++rc) {
                const int rs = rc % GEMM_NRAW;
                if (rc >= GEMM_NRAW && !mbar_wait_sleep(&raw_empty[rs], ((rc / GEMM_NRAW) - 1) & 1, 100)) {
                    if (lane == 0) atomicExch(p.err, 8);
                    alive = false;
                    break;
                }
                const uint32_t dst = smem_u32(raw_base) + rs * RAW_SLOT;
                // G tiled copies per half tile: copy j brings, for each of the 128 / G row groups, the window
                // of PITCH bytes that holds block b of the group's row j (it starts on the 16-byte boundary at or
                // below the block; bytes past the end of a group arrive as zeros and are never read)
                const int G = 1 << p.g_log2;
                if (lane == 0) mbar_arrive_expect_tx(&raw_full[rs], (uint32_t)((two ? 2 : 1) * RAW_HALF));
                __syncwarp();
                if (lane < 2 * G && (lane < G || two)) {
                    const int h = lane >= G, j = lane & (G - 1);
                    const int x = (j * p.rb + b * BB) & ~15;
                    const int row0 = (DUAL || h == 0) ? m0 : m0 + GEMM_BM;
                    tma_load_3d(dst + h * RAW_HALF + j * (GEMM_BM >> p.g_log2) * PITCH, &maps.wmap[DUAL ? h : 0], x,
                                row0 >> p.g_log2, e, &raw_full[rs]);
                }
                __syncwarp();
            }
        }
    } else if (warp == 2) {
        // ------------------------------- activation loader ------------------------------------
        int it = 0;
        for (int tile = blockIdx.x; tile < n_tiles && alive; tile += gridDim.x) {
            int e, m0, p0, np;
            tile_info(tile, e, m0, p0, np);
            const int bi = (np + 31) / 32 - 1;       // the smallest box that covers the tile's pairs
            for (int ks = 0; ks < ksteps; ++ks, ++it) {
                const int sb = it % GEMM_NB;
                if (!mbar_wait_sleep(&done[sb], ((it / GEMM_NB) - 1) & 1, 100)) {
                    if (lane == 0) atomicExch(p.err, 10);
                    alive = false;
                    break;
                }
                if (lane == 0) {
                    // rows p0 .. of the sorted activations, 64 columns; rows past the end of the buffer arrive as zeros
                    mbar_arrive_expect_tx(&in_full[sb], (uint32_t)(32 * (bi + 1) * GEMM_BK * 2));
                    // the k of the four steps of a super-block: 0, 128, 64, 192 (the converters' groups take a half each, in turn)
                    const int k64 = (ks & ~3) | ((ks & 1) << 1) | ((ks >> 1) & 1);
                    tma_load_2d(smem + sb * B_BYTES, &maps.box[bi], k64 * GEMM_BK, p0, &in_full[sb]);
                }
                __syncwarp();
            }
        }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, TMEM_COLS);
}

}  // namespace zmoe
