// Large-batch ("prefill") expert FFN: grouped GEMMs on the 5th-generation tensor cores.
//
// Orientation: the WEIGHTS are the M operand (128 output features per tile) and the expert's
// token rows are the N operand (up to 192 per tile, any multiple of 16), so ragged expert
// groups cost at most 15 padded rows instead of a padded 128-row tile.  D (FP32) lives in
// tensor memory: lane = output feature, column = token.
//
//   warp 0        TMA producer: activation tiles [N x 64] f16 -> shared memory (128-byte swizzle)
//   warps 1, 3    MMA issuers: the warp walks its loop converged and one elected lane issues tcgen05.mma
//                 (kind::f16, M=128, K=16), warp 1 for the first weight tile of a stage, warp 3 for the second.
//                 An issuer is serial (barrier polls, commits) and the tensor pipe drains whenever it is not
//                 issuing; two issuers cover each other's gaps
//   warp 2        TMA producer for the packed 4-bit weights: [128 rows x 128 B] blocks (256 columns)
//                 land in a 128-byte-swizzled staging ring
//   warps 4..19   decoders: each lane owns one weight row (= one tensor-memory lane), reads 32 packed
//                 bytes (64 columns) of it per turn from the staging area, decodes exactly
//                 to f16 (hardware E2M1 conversion / INT4 magic-number trick), applies the block
//                 scale and writes the 32 f16x2 words straight into TENSOR MEMORY (tcgen05.st):
//                 the decoded weights are the A operand of a tensor-memory-sourced MMA and never
//                 touch shared memory, which halves the shared-memory traffic per MMA
//   warps 20..27  epilogue: tcgen05.ld the accumulators, fuse SwiGLU (gate/up) or the output
//                 scale (down), store
// Tensor memory (512 columns): the accumulators (two tiles x NT tokens, two sets of them for small tiles), behind them
// the ring of decoded weight slices (see Geo).  BF16 weights (the shared expert, BF16 experts) need no decode and keep
// the shared-memory A operand.
// CTAs are persistent (one per SM) and walk a tile list built on the device from the
// per-expert offsets.
//
// Every wait is bounded: on expiry the kernel raises kStatusWaitTimeout, all roles leave their
// loops, tensor memory is released and the kernel returns normally.
//
// Replaces the reference's per-row page kernels (kernels/cuda/backend.cu:2439-2582, 2600-2779)
// and the per-expert matmul fallbacks (kernels/cuda/backend.cu:1140-1207).
#include <cuda.h>
#include <cuda_fp16.h>

#include <cstddef>
#include <cstdlib>

#include "common.cuh"
#include "tc5.cuh"

namespace smoe {

// Tokens per tile NT: 192 (an expert with up to 192 rows is decoded once) when groups are large, 160 for groups of
// about 128 rows, 128 and below when they are small.  A stage is kKst columns of K: the roles hand a stage over through
// barriers, and one hand-over (two waits, the MMAs, two commits) costs the issuing thread 400 to 700 clocks whatever
// the stage holds, which set the pace of tiles of up to 128 tokens at 64 columns; with 192 or 160 tokens the MMAs of
// 64 columns take longer than that and tensor memory has no room for more.
template <int NT>
struct Geo {
    static_assert(NT == 32 || NT == 64 || NT == 128 || NT == 160 || NT == 192, "tile sizes");
    static constexpr uint32_t kNTile = NT;
    static constexpr uint32_t kKst = NT <= 128 ? 128u : 64u;
    static constexpr uint32_t kAccBufs = NT <= 64 ? 2u : 1u;                       // accumulator sets: the epilogue of a tile beside the next main loop
    static constexpr uint32_t kAccCols = kAccBufs * 2u * NT;                       // accumulator columns (2 tiles x NT each)
    static constexpr uint32_t kAStageCols = kKst;                                  // tensor-memory columns per A stage: 2 tiles x kKst / 2
    static constexpr uint32_t kAStages = (512u - kAccCols) / kAStageCols;          // tensor-memory ring of decoded weight slices
    static constexpr uint32_t kBTile = NT * kKst * 2u;                             // bytes of one activation stage
    static constexpr uint32_t kBStages = NT <= 64 ? 4u : NT == 128 ? 3u : 6u;      // activation stages in flight
    static constexpr uint32_t kPkBufs = NT == 32 ? 6u : NT == 64 ? 5u : NT == 128 ? 4u : NT == 160 ? 3u : 2u;
};
constexpr uint32_t kMaxStages = 8;   // barriers per ring
constexpr uint32_t kMTile = 128;    // output features per tile
constexpr uint32_t kBK = 64;        // columns of one 128-byte swizzled row: the unit of TMA boxes and of a decode turn
constexpr uint32_t kATile = kMTile * kBK * 2;  // 16 KiB: 128 weight rows x 64 columns of 16 bits
constexpr uint32_t kDecodeWarps = 16;  // a lane decodes 64 columns of one row per turn
constexpr uint32_t kEpilogueWarps = 8;   // two per tensor-memory lane quarter: even / odd 16-token chunks
constexpr uint32_t kThreads = (4 + kDecodeWarps + kEpilogueWarps) * 32;
constexpr uint32_t kPkCols = 256;                       // columns per packed staging block (four 64-column slabs)
constexpr uint32_t kPkTile = kMTile * (kPkCols / 2);    // 16 KiB of 4-bit weights: 128 rows x 128 B
constexpr uint32_t kFirstDecodeWarp = 4, kFirstEpilogueWarp = kFirstDecodeWarp + kDecodeWarps;
constexpr uint32_t kMinTileRows = 16;   // token rows of the smallest tile: bounds the tile list
constexpr int kFmtInt4N = 4;    // INT4 whose scales span at most six octaves per projection (see p_int4x8_narrow)
constexpr int kFmtBf16W = 3;  // plain BF16 weights (shared expert): tiles arrive by TMA, no decode

// ------------------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ bool epilogue_vote(bool failed) { return group_vote<kEpilogueWarps * 32u>(failed); }
// Instruction descriptor, kind::f16: F16 x F16 (or BF16 x BF16) -> F32, both operands K-major, M = 128.
__device__ __forceinline__ uint32_t umma_idesc_f16(uint32_t n, uint32_t ab_format /* 0 = F16, 1 = BF16 */) {
    uint32_t d = 0;
    d |= 1u << 4;               // D format F32
    d |= ab_format << 7;        // A format
    d |= ab_format << 10;       // B format
    d |= (n >> 3) << 17;        // N
    d |= (kMTile >> 4) << 24;   // M
    return d;
}
// The four K = 16 MMAs of one 64-column slab, A from tensor memory (lane = row, 32-bit column = two K values, 8 columns
// per MMA) or from shared memory; the low words of the shared-memory descriptors come in, the high word is constant.
//
// Two things decide what an MMA costs the issuing warp.  (1) Its operands live in uniform registers: the warp runs its
// loop converged, with values the compiler can prove uniform, and only the MMA itself is left to one elected lane.  With
// one lane in a divergent branch and operands in ordinary registers an issue took 80 to 140 clocks, so that the issuers
// were busy for 75 % of the kernel's time and set its pace.  (2) MMAs that follow one another in straight-line code ran
// without overlap (512 MMAs of 128 x N x 16, clocks per MMA: A in tensor memory 74 / 106 at N = 128 / 192, A in shared
// memory 107 / 139); with a branch between them they pipeline (64 / 96, the tensor pipe's rate).  `never` is a value the
// compiler cannot see through that is never 0: the branches on it are not taken and only end the basic blocks.
__device__ __forceinline__ void umma4_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t idesc,
                                             uint32_t accumulate, uint32_t never) {
    asm volatile(
        "{\n .reg .pred p, t, q;\n .reg .b64 b0, b1, b2, b3;\n .reg .b32 a1, a2, a3, l1, l2, l3;\n"
        " setp.ne.b32 p, %4, 0;\n setp.eq.b32 t, 0, 0;\n setp.eq.b32 q, %5, 0;\n"
        " add.u32 l1, %2, 2;\n add.u32 l2, %2, 4;\n add.u32 l3, %2, 6;\n"
        " mov.b64 b0, {%2, %6};\n mov.b64 b1, {l1, %6};\n mov.b64 b2, {l2, %6};\n mov.b64 b3, {l3, %6};\n"
        " add.u32 a1, %1, 8;\n add.u32 a2, %1, 16;\n add.u32 a3, %1, 24;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b0, %3, p;\n @q bra DONE;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, t;\n @q bra DONE;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, t;\n @q bra DONE;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, t;\n DONE:\n}" ::"r"(tmem_d),
        "r"(tmem_a), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(never), "n"(kDescHi)
        : "memory");
}
__device__ __forceinline__ void umma4_f16_ss(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                             uint32_t accumulate, uint32_t never) {
    asm volatile(
        "{\n .reg .pred p, t, q;\n .reg .b64 a0, a1, a2, a3, b0, b1, b2, b3;\n .reg .b32 k1, k2, k3, l1, l2, l3;\n"
        " setp.ne.b32 p, %4, 0;\n setp.eq.b32 t, 0, 0;\n setp.eq.b32 q, %5, 0;\n"
        " add.u32 l1, %2, 2;\n add.u32 l2, %2, 4;\n add.u32 l3, %2, 6;\n"
        " add.u32 k1, %1, 2;\n add.u32 k2, %1, 4;\n add.u32 k3, %1, 6;\n"
        " mov.b64 b0, {%2, %6};\n mov.b64 b1, {l1, %6};\n mov.b64 b2, {l2, %6};\n mov.b64 b3, {l3, %6};\n"
        " mov.b64 a0, {%1, %6};\n mov.b64 a1, {k1, %6};\n mov.b64 a2, {k2, %6};\n mov.b64 a3, {k3, %6};\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], a0, b0, %3, p;\n @q bra DONE;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %3, t;\n @q bra DONE;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, %3, t;\n @q bra DONE;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], a3, b3, %3, t;\n DONE:\n}" ::"r"(tmem_d),
        "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(never), "n"(kDescHi)
        : "memory");
}
// ------------------------------------------------------------------------------ decoders (f16)
__device__ __forceinline__ void p_e2m1x8_f16(uint32_t w, uint32_t r[4]) {
    asm("{\n .reg .b8 b0, b1, b2, b3;\n mov.b32 {b0, b1, b2, b3}, %4;\n"
        " cvt.rn.f16x2.e2m1x2 %0, b0;\n cvt.rn.f16x2.e2m1x2 %1, b1;\n"
        " cvt.rn.f16x2.e2m1x2 %2, b2;\n cvt.rn.f16x2.e2m1x2 %3, b3;\n}"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
        : "r"(w));
}
__device__ __forceinline__ uint32_t p_mul_f16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t p_fma_f16x2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t p_sub_f16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
// 8 offset-binary INT4 nibbles -> 4 f16x2 of (q - 8), register i = columns i and i + 4 (the activation rows are stored
// in that order, see int4_slot).  Four nibbles of a word land in the low bits of 0x6400 halves with one logic
// instruction each: 0x6400 | q is the f16 number 1024 + q, 0x6400 | 16 q is 1024 + 16 q, and one packed add or
// multiply-add leaves q - 8 exactly.  9 instructions for 8 weights; the natural column order took 13.
__device__ __forceinline__ uint32_t p_magic(uint32_t w, uint32_t mask) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(w), "r"(mask), "r"(0x64006400u));   // (w & mask) | 0x64006400
    return d;
}
__device__ __forceinline__ void p_int4x8_f16(uint32_t w, uint32_t r[4]) {
    const uint32_t w8 = w >> 8;
    const uint32_t k1032 = 0x64086408u, k16th = 0x2C002C00u, km72 = 0xD480D480u;   // 1032, 1 / 16, -72
    r[0] = p_sub_f16x2(p_magic(w, 0x000F000Fu), k1032);
    r[1] = p_fma_f16x2(p_magic(w, 0x00F000F0u), k16th, km72);
    r[2] = p_sub_f16x2(p_magic(w8, 0x000F000Fu), k1032);
    r[3] = p_fma_f16x2(p_magic(w8, 0x00F000F0u), k16th, km72);
}
// The same weights times their scale in ONE multiply-add per pair, 9 instructions for 8 weights where the above and the
// multiplication by the scale take 13.  A nibble that a mask leaves in the low bits of a half is the subnormal f16 number
// n 2^-24, or n 2^-20 four bits higher; with m24 = 2^24 s, m20 = 2^20 s and c = -8 s the multiply-add is (n - 8) s, exact:
// its result has at most eleven significant bits.  2^24 s has to stay below 2^16, and s at or above 2^-14 keeps the products
// normal numbers (of subnormal ones the MMA keeps fewer bits), so the scales of a projection, times a power of two of its own
// (WeightTable::emin holds 2^24 of it as a float, post_scale undoes it), lie in [2^-14, 2^-8): six octaves, and the bits of the
// result are those of the decode above.  6144 x 2048 x 256 experts, whole layer, in turn: 4 tokens 240 -> 222 us, 333 tokens
// 1436 -> 1349, 4096 tokens 2559 -> 2514 (2909 -> 2859 once the power cap holds the clock).
__device__ __forceinline__ void p_int4x8_narrow(uint32_t w, uint32_t m24, uint32_t m20, uint32_t c, uint32_t r[4]) {
    const uint32_t w8 = w >> 8;
    r[0] = p_fma_f16x2(w & 0x000F000Fu, m24, c);
    r[1] = p_fma_f16x2(w & 0x00F000F0u, m20, c);
    r[2] = p_fma_f16x2(w8 & 0x000F000Fu, m24, c);
    r[3] = p_fma_f16x2(w8 & 0x00F000F0u, m20, c);
}
// Pins 32 computed registers before whatever follows.
__device__ __forceinline__ void keep32(const uint32_t v[32]) {
#pragma unroll
    for (int i = 0; i < 32; i += 16)
        asm volatile("" ::"r"(v[i]), "r"(v[i + 1]), "r"(v[i + 2]), "r"(v[i + 3]), "r"(v[i + 4]), "r"(v[i + 5]), "r"(v[i + 6]),
                     "r"(v[i + 7]), "r"(v[i + 8]), "r"(v[i + 9]), "r"(v[i + 10]), "r"(v[i + 11]), "r"(v[i + 12]), "r"(v[i + 13]),
                     "r"(v[i + 14]), "r"(v[i + 15]));
}

// Activation tensor maps with boxes of 16, 32, 64 and 128 rows: a tile with few valid rows
// fetches only the rows the MMA will read (rounded up to the next box size).
struct BMaps {
    CUtensorMap m[4];
};

struct TileInfo {
    uint32_t g, row0, n;  // expert, first row of this n-tile, valid rows (1..kNTile)
    uint32_t m0;          // first output feature
};

template <int NT>
struct __align__(1024) PrefillSmem {
    // 4-bit formats: packed staging [buffer][gate/down, up][kPkTile], then the activation ring.
    // BF16 weights: w and b together are one arena that the kernel cuts into stages of A tiles
    // [stage][gate/down, up][64-column slab][kATile] followed by the activation stages that still fit.
    uint8_t w[Geo<NT>::kPkBufs][2][kPkTile];
    uint8_t b[Geo<NT>::kBStages][Geo<NT>::kBTile];   // activation stages: [slab of 64 columns][NT rows][128 B]
    uint64_t full_a[kMaxStages], empty_a[kMaxStages], full_b[kMaxStages], empty_b[kMaxStages];
    uint64_t pk_full[Geo<NT>::kPkBufs], pk_empty[Geo<NT>::kPkBufs];
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    uint32_t abort_flag;
};

__device__ __forceinline__ bool tile_lookup(const PrefillArgs& a, uint32_t tile, uint32_t total, uint32_t m_tiles, TileInfo& t,
                                            uint32_t tile_feat) {
    if (tile >= total) return false;
    const uint32_t j = tile / m_tiles;
    if (a.tile_table) {
        t.g = a.tile_table[4 + 3 * j];
        t.row0 = a.tile_table[4 + 3 * j + 1];
        t.n = a.tile_table[4 + 3 * j + 2];
    } else {
        t.g = 0;
        t.row0 = j * a.ntile;
        t.n = min(a.ntile, a.pairs - t.row0);
    }
    t.m0 = a.feat0 + (tile - j * m_tiles) * tile_feat;
    return true;
}

// Position of an activation column in the rows the INT4 tiles multiply: the decoder leaves the nibbles of a weight
// word as the pairs (0,4) (1,5) (2,6) (3,7), so columns i and i + 4 of every eight lie side by side.
__device__ __forceinline__ uint32_t int4_slot(uint32_t c) {
    const uint32_t p = c & 7u;
    return (c & ~7u) | ((p & 3u) << 1) | (p >> 2);
}

// MODE 0: gate + up tiles of the same 128 features, SwiGLU, act (16-bit) out.  K = H, features over I.
// MODE 1: one down tile (128 features), y (fp32) out.                          K = I, features over H.
// MODE 2: two adjacent down tiles (256 features) against the same activation tile -- halves the
//         shared-memory traffic per MMA of MODE 1; needs H % 256 == 0.
// DUAL (two weight tiles and two accumulators per activation tile) = MODE 0 or 2.
// SPLIT: the activation is a 16-bit hi + lo pair; a stage holds the hi rows and behind them the lo rows, one MMA
// multiplies both and the epilogue adds the two halves of the accumulator columns, so a tile holds NT / 2 tokens.
template <int FMT, int MODE, int NT, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1)
prefill_ffn_kernel(const __grid_constant__ BMaps maps_b, const __grid_constant__ BMaps maps_lo,
                   const __grid_constant__ CUtensorMap map_a0, const __grid_constant__ CUtensorMap map_a1, PrefillArgs a,
                   const float* __restrict__ rowscale, void* __restrict__ act_out_v,
                   const CUtensorMap* __restrict__ wmaps /* [3][n_groups] */) {
    extern __shared__ uint8_t smem_raw[];
    using G = Geo<NT>;
    PrefillSmem<NT>& S =
        *reinterpret_cast<PrefillSmem<NT>*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr bool DUAL = MODE != 1;
    constexpr bool GU = MODE == 0;
    constexpr bool BF = FMT == kFmtBf16W;
    constexpr uint32_t kKst = G::kKst, kSlabs = kKst / kBK;
    constexpr uint32_t kAccCols = G::kAccCols, kAccBufs = G::kAccBufs, kPkBufs = G::kPkBufs;
    // BF16 weights arrive as ready A tiles by TMA: the staging blocks and the activation ring are re-cut into stages
    // of weight tiles and as many activation stages as the rest holds
    constexpr uint32_t kArena = kPkBufs * 2u * kPkTile + G::kBStages * G::kBTile;
    constexpr uint32_t kBfATile = kSlabs * kATile;                       // one weight tile of a stage
    constexpr uint32_t kBfAStage = (DUAL ? 2u : 1u) * kBfATile;
    constexpr uint32_t kBfAWant = (NT <= 64 ? 192u : 128u) * 1024u / kBfAStage;
    constexpr uint32_t kBfAStages = kBfAWant < kMaxStages ? kBfAWant : kMaxStages;
    constexpr uint32_t kBfBFit = (kArena - kBfAStages * kBfAStage) / G::kBTile;
    constexpr uint32_t kAStages = BF ? kBfAStages : G::kAStages;
    constexpr uint32_t kBStages = BF ? (kBfBFit < kMaxStages ? kBfBFit : kMaxStages) : G::kBStages;
    static_assert(kAStages >= 2u && kAStages <= kMaxStages && kBStages >= 2u && kBStages <= kMaxStages, "ring geometry");
    static_assert(offsetof(PrefillSmem<NT>, b) == kPkBufs * 2u * kPkTile, "staging blocks and activation ring form one arena");
    uint8_t* const arena = &S.w[0][0][0];
    uint8_t* const b_base = BF ? arena + kBfAStages * kBfAStage : &S.b[0][0];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    constexpr uint32_t kTileFeat = MODE == 2 ? 2u * kMTile : kMTile;  // features per tile
    constexpr uint32_t kSecond = MODE == 2 ? kMTile : 0u;              // row offset of the second weight tile
    const uint32_t K = GU ? a.H : a.I;
    const uint32_t R = GU ? a.I : a.H;
    const uint32_t m_tiles = (!GU && a.feats ? a.feats : R) / kTileFeat;
    const uint32_t k_stages = K / kKst;
    volatile uint32_t* abort_flag = &S.abort_flag;
    const uint32_t total = (a.tile_table ? a.tile_table[0] : (a.pairs + a.ntile - 1u) / a.ntile) * m_tiles;
    if (total == 0u) return;   // no rows (a rank that received none): leave before any set-up

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kMaxStages; ++s) {
            // one arrival per decode warp that fills part of the stage (a 64-column stage is decoded by half of the
            // decode warps, the other half works on the next one), or one TMA transaction group for BF16 weights
            mbar_init(&S.full_a[s], BF ? 1u : kDecodeWarps / (kSlabs == 1u ? 2u : 1u) / (DUAL ? 1u : 2u));
            mbar_init(&S.empty_a[s], DUAL ? 2u : 1u);   // one commit per MMA issuer
            mbar_init(&S.full_b[s], 1);
            mbar_init(&S.empty_b[s], DUAL ? 2u : 1u);
        }
        for (uint32_t i = 0; i < 2u; ++i) {
            mbar_init(&S.acc_full[i], DUAL ? 2u : 1u);
            mbar_init(&S.acc_empty[i], kEpilogueWarps);  // one arrival per epilogue warp
        }
        for (uint32_t i = 0; i < kPkBufs; ++i) {
            mbar_init(&S.pk_full[i], 1);
            mbar_init(&S.pk_empty[i], DUAL ? kDecodeWarps : kDecodeWarps / 2u);
        }
        S.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {  // tensor-memory allocation: all 512 columns (one CTA per SM)
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem_base)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = S.tmem_base;
    // rows of the box that fetches n activation rows (boxes of 16, 32, 64 and 128 rows exist)
    auto box_of = [](uint32_t n) { return n <= 16u ? 0u : (n <= 32u ? 1u : (n <= 64u ? 2u : 3u)); };

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer: activation rows
        if (lane == 0) {
            uint32_t issued = 0;
            Ring<kBStages> rb;
            bool ok = true;
            TileInfo t, tn;
            bool have = tile_lookup(a, blockIdx.x, total, m_tiles, t, kTileFeat);
            for (uint32_t tile = blockIdx.x; ok && have; tile += gridDim.x) {
                const bool hn = tile_lookup(a, tile + gridDim.x, total, m_tiles, tn, kTileFeat);
                const uint32_t bsel = box_of(t.n), rows = 16u << bsel;
                const bool tail = NT > 128 && t.n > 128u;   // rows from 128 on arrive as a second box: 64 rows (192-token tile) or 32
                constexpr uint32_t kTailSel = NT == 192 ? 2u : 1u, kTailRows = 16u << kTailSel;
                const uint32_t bytes = (rows * (SPLIT ? 2u : 1u) + (tail ? kTailRows : 0u)) * kKst * 2u;
                for (uint32_t ks = 0; ks < k_stages; ++ks) {
                    if (!mbar_wait(&S.empty_b[rb.i], rb.ph ^ 1u, abort_flag)) { ok = false; break; }
                    mbar_arrive_expect_tx(&S.full_b[rb.i], bytes);
                    uint8_t* dst = b_base + rb.i * G::kBTile;
#pragma unroll
                    for (uint32_t h = 0; h < kSlabs; ++h) {
                        const uint32_t x = ks * kKst + h * kBK;
                        tma_load_2d(dst + h * (NT * 128u), &maps_b.m[bsel], x, t.row0, &S.full_b[rb.i]);
                        if (SPLIT) tma_load_2d(dst + h * (NT * 128u) + rows * 128u, &maps_lo.m[bsel], x, t.row0, &S.full_b[rb.i]);
                        if (tail) tma_load_2d(dst + h * (NT * 128u) + 128u * 128u, &maps_b.m[kTailSel], x, t.row0 + 128u, &S.full_b[rb.i]);
                    }
                    ++issued;
                    rb.next();
                }
                t = tn;
                have = hn;
            }
            if (!ok) { *abort_flag = 1; atomicOr(a.status, kStatusWaitTimeout); }
            if (*abort_flag) drain_copies(S.full_b, issued, kBStages);
        }
    } else if (warp == 1 || warp == 3) {
        // ---------------------------------------------------------------- MMA issuers
        const uint32_t mi = warp == 3 ? 1u : 0u;   // which weight tile of the stage this warp feeds
        if (DUAL || mi == 0u) {
            // the whole warp walks the loop (see umma4_f16_ts): every loop condition is a vote or comes from lane 0
            auto uni = [](uint32_t v) { return __shfl_sync(0xFFFFFFFFu, v, 0); };
            auto all = [](bool b) { return __all_sync(0xFFFFFFFFu, b); };
            const bool el = elect_one();
            const uint32_t tm = uni(tmem_base), tiles = uni(total);
            Ring<kAStages> ra;
            Ring<kBStages> rb;
            Ring<kAccBufs> rc;
            const uint32_t b_lo0 = umma_desc_lo(smem_u32(b_base));
            const uint32_t a_lo0 = umma_desc_lo(smem_u32(arena) + mi * kBfATile);
            bool ok = true;
            TileInfo t, tn;
            tile_lookup(a, blockIdx.x, total, m_tiles, t, kTileFeat);
            for (uint32_t tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
                tile_lookup(a, tile + gridDim.x, total, m_tiles, tn, kTileFeat);
                const uint32_t rows = uni(t.n);
                if (!all(mbar_wait(&S.acc_empty[rc.i], rc.ph ^ 1u, abort_flag))) { ok = false; break; }
                tc_fence_after();
                const uint32_t n = SPLIT ? 32u << box_of(rows) : (rows + 15u) & ~15u;
                const uint32_t idesc = umma_idesc_f16(n, BF ? 1u : 0u);
                const uint32_t d = tm + rc.i * (2u * NT) + mi * NT;
                for (uint32_t ks = 0; ks < k_stages; ++ks) {
                    const bool got = mbar_wait(&S.full_a[ra.i], ra.ph, abort_flag) && mbar_wait(&S.full_b[rb.i], rb.ph, abort_flag);
                    if (!all(got)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t b_lo = b_lo0 + rb.i * (G::kBTile >> 4);
                    const uint32_t a_lo = a_lo0 + ra.i * (kBfAStage >> 4);
                    const uint32_t ta = tm + kAccCols + ra.i * G::kAStageCols + mi * (kKst / 2u);
                    if (el) {
#pragma unroll
                        for (uint32_t h = 0; h < kSlabs; ++h) {
                            if (BF) umma4_f16_ss(d, a_lo + h * (kATile >> 4), b_lo + h * (NT * 128u >> 4), idesc, h ? 1u : ks, a.H);
                            else umma4_f16_ts(d, ta + h * (kBK / 2u), b_lo + h * (NT * 128u >> 4), idesc, h ? 1u : ks, a.H);
                        }
                        umma_commit(&S.empty_a[ra.i]);  // a stage is free once both issuers' MMAs have read it
                        umma_commit(&S.empty_b[rb.i]);
                    }
                    __syncwarp();
                    ra.next();
                    rb.next();
                }
                if (ok && el) umma_commit(&S.acc_full[rc.i]);
                __syncwarp();
                rc.next();
                t = tn;
            }
            if (!ok && lane == 0) { *abort_flag = 1; atomicOr(a.status, kStatusWaitTimeout); }
        }
    } else if (warp == 2) {
        // ---------------------------------------------------------------- TMA producer: weights
        if (lane == 0) {
            uint32_t issued = 0;
            bool ok = true;
            TileInfo t, tn;
            Ring<BF ? kAStages : kPkBufs> rw;
            const uint32_t blocks = BF ? k_stages : (K + kPkCols - 1u) / kPkCols;
            bool have = tile_lookup(a, blockIdx.x, total, m_tiles, t, kTileFeat);
            for (uint32_t tile = blockIdx.x; ok && have; tile += gridDim.x) {
                const bool hn = tile_lookup(a, tile + gridDim.x, total, m_tiles, tn, kTileFeat);
                // BF16: a map per expert when there is a table, else the one matrix pair of the launch
                const CUtensorMap* m0 = BF && !wmaps ? &map_a0 : wmaps + (GU ? 0u : 2u) * a.n_groups + t.g;
                const CUtensorMap* m1 = BF && !wmaps ? &map_a1 : wmaps + (GU ? 1u : 2u) * a.n_groups + t.g;
                for (uint32_t q = 0; q < blocks; ++q) {
                    uint64_t* full = BF ? &S.full_a[rw.i] : &S.pk_full[rw.i % kPkBufs];
                    uint64_t* empty = BF ? &S.empty_a[rw.i] : &S.pk_empty[rw.i % kPkBufs];
                    if (!mbar_wait(empty, rw.ph ^ 1u, abort_flag)) { ok = false; break; }
                    if (BF) {
                        mbar_arrive_expect_tx(full, kBfAStage);
                        uint8_t* dst = arena + rw.i * kBfAStage;
#pragma unroll
                        for (uint32_t h = 0; h < kSlabs; ++h) {
                            tma_load_2d(dst + h * kATile, m0, q * kKst + h * kBK, t.m0, full);
                            if (DUAL) tma_load_2d(dst + kBfATile + h * kATile, m1, q * kKst + h * kBK, t.m0 + kSecond, full);
                        }
                    } else {
                        mbar_arrive_expect_tx(full, DUAL ? 2u * kPkTile : kPkTile);
                        uint8_t* dst = arena + rw.i * (2u * kPkTile);
                        tma_load_2d(dst, m0, q * (kPkCols / 2u), t.m0, full);
                        if (DUAL) tma_load_2d(dst + kPkTile, m1, q * (kPkCols / 2u), t.m0 + kSecond, full);
                    }
                    ++issued;
                    rw.next();
                }
                t = tn;
                have = hn;
            }
            if (!ok) { *abort_flag = 1; atomicOr(a.status, kStatusWaitTimeout); }
            if (*abort_flag) {
                if (BF) drain_copies(S.full_a, issued, kAStages);
                else drain_copies(S.pk_full, issued, kPkBufs);
            }
        }
    } else if (warp < kFirstEpilogueWarp && BF) {
        // BF16 weights need no decode: the TMA producer loads their tiles
    } else if (warp < kFirstEpilogueWarp) {
        // ---------------------------------------------------------------- weight decoders
        // A warp can only write the tensor-memory lanes 32 * (warp % 4) .. + 31, and a lane holds one weight row:
        // lane i of a decode warp owns row 32 * (warp % 4) + i of one weight tile.  The four decode warps that share
        // a lane quarter split into tile 0 / tile 1 and even / odd 64-column slabs: a warp takes every other slab,
        // decodes it into 32 registers BEFORE it waits for the slab's place in tensor memory (the decode then
        // overlaps the MMAs that still read that place), stores, and hands over.  (32 consecutive rows reading the
        // same swizzled 16-byte chunk index are free of bank conflicts.)  With one weight tile per stage (MODE 1)
        // only the tile-0 warps work.
        const uint32_t wd = warp - kFirstDecodeWarp;
        const uint32_t which = DUAL ? (wd >> 3) : 0u;
        const uint32_t sub = (wd >> 2) & 1u;
        const uint32_t arow = (warp & 3u) * 32u + lane;
        const uint32_t a_lane = tmem_base + (((warp & 3u) * 32u) << 16) + kAccCols + which * (kKst / 2u) +
                                (kSlabs == 2u ? sub * (kBK / 2u) : 0u);
        const uint32_t off0 = ((2u * sub) ^ (arow & 7u)) << 4, off1 = off0 ^ 16u;   // this warp's first slab; the other is ^ 64
        constexpr bool kEmin = FMT == STRATA_MOE_FMT_MXFP4 || FMT == kFmtInt4N;
        const WeightTable& wt = GU ? (which ? a.up : a.gate) : a.down;
        const uint32_t blocks = (K + kPkCols - 1u) / kPkCols, k_slabs = K / kBK;
        const size_t scale_row = FMT == STRATA_MOE_FMT_MXFP4 ? K / 32u : FMT == STRATA_MOE_FMT_NVFP4 ? K / 16u : K / 128u * 2u;
        // Scale bytes of one 256-column block of a row: MXFP4 8 bytes, NVFP4 16 bytes, INT4 two BF16 values.  Vector
        // loads need rows of whole blocks (K % 256 == 0); the last block of other rows takes narrow loads.
        const bool whole_blocks = (K % kPkCols) == 0u;
        auto load_scales = [&](const uint8_t* srow, uint32_t q) -> uint4 {
            uint4 v = make_uint4(0, 0, 0, 0);
            if (FMT == STRATA_MOE_FMT_MXFP4) {          // 8 bytes per block, rows 4-byte aligned
                if (whole_blocks) {
                    const uint2 w = __ldg(reinterpret_cast<const uint2*>(srow + q * 8u));
                    v.x = w.x; v.y = w.y;
                } else {
                    v.x = __ldg(reinterpret_cast<const uint32_t*>(srow + q * 8u));
                    if ((q + 1u) * 8u <= K / 32u) v.y = __ldg(reinterpret_cast<const uint32_t*>(srow + q * 8u + 4u));
                }
            } else if (FMT == STRATA_MOE_FMT_NVFP4) {   // 16 bytes per block, rows 8-byte aligned
                if (whole_blocks) {
                    v = __ldg(reinterpret_cast<const uint4*>(srow + q * 16u));
                } else {
                    const uint2 w = __ldg(reinterpret_cast<const uint2*>(srow + q * 16u));
                    v.x = w.x; v.y = w.y;
                    if ((q + 1u) * 16u <= K / 16u) {
                        const uint2 w2 = __ldg(reinterpret_cast<const uint2*>(srow + q * 16u + 8u));
                        v.z = w2.x; v.w = w2.y;
                    }
                }
            } else {                                     // two BF16 per block, rows 2-byte aligned
                if (whole_blocks) {
                    v.x = __ldg(reinterpret_cast<const uint32_t*>(srow + q * 4u));
                } else {
                    v.x = __ldg(reinterpret_cast<const unsigned short*>(srow + q * 4u));
                    if ((q + 1u) * 2u <= K / 128u)
                        v.x |= (uint32_t)__ldg(reinterpret_cast<const unsigned short*>(srow + q * 4u + 2u)) << 16;
                }
            }
            return v;
        };
        Ring<kAStages> ra;
        if (kSlabs == 1u) ra.i = sub;      // 64-column stages: this warp fills every other one
        Ring<kPkBufs> rp;
        bool ok = true;
        TileInfo t, tn;
        bool have = (DUAL || wd < kDecodeWarps / 2u) && tile_lookup(a, blockIdx.x, total, m_tiles, t, kTileFeat);
        const uint8_t *srow = nullptr, *sbase = nullptr;
        uint32_t emin = 0;      // MXFP4: smallest scale byte; narrow INT4: the float its scales are multiplied by
        uint4 sc_next = make_uint4(0, 0, 0, 0);
        if (have) {
            srow = wt.scales[t.g] + (t.m0 + arow + which * kSecond) * scale_row;
            if (kEmin) emin = wt.emin[t.g];
            sc_next = load_scales(srow, 0);
        }
        for (uint32_t tile = blockIdx.x; ok && have; tile += gridDim.x) {
            // the next tile's entry, scale base and first scales are requested one step before they are needed: a chain of
            // dependent loads at every tile start would stop the decoders for about a thousand clocks
            const bool hn = tile_lookup(a, tile + gridDim.x, total, m_tiles, tn, kTileFeat);
            uint32_t emin_n = 0;
            const uint32_t mx_add = (uint32_t)(2 - (int32_t)emin) * 0x04000400u;
            for (uint32_t q = 0; q < blocks; ++q) {
                const uint4 sc = sc_next;
                if (q + 1u < blocks) sc_next = load_scales(srow, q + 1u);
                else if (hn && blocks > 1u) sc_next = load_scales(srow, 0);     // the next tile's row by now
                if (!mbar_wait_warp(&S.pk_full[rp.i], rp.ph, abort_flag)) { ok = false; break; }
                const uint8_t* pk_row = arena + (rp.i * 2u + which) * kPkTile + arow * 128u;
                const uint32_t sel[2] = {FMT == STRATA_MOE_FMT_NVFP4 ? (sub ? sc.y : sc.x) : sc.x,
                                         FMT == STRATA_MOE_FMT_NVFP4 ? (sub ? sc.w : sc.z)
                                                                     : (FMT == STRATA_MOE_FMT_MXFP4 ? sc.y : sc.x >> 16)};
#pragma unroll
                for (uint32_t jj = 0; jj < 2u; ++jj) {
                    if (q * 4u + jj * 2u >= k_slabs) break;   // K % 256 == 128: the last block holds two slabs
                    uint32_t v[32];
                    uint32_t m24 = 0, m20 = 0, mc = 0;
                    if (FMT == kFmtInt4N) {
                        // one scale for the slab's 64 columns; powers of two are steps of the exponent field (a zero stays zero)
                        const float sf = __uint_as_float(sel[jj] << 16) * __uint_as_float(emin);
                        m24 = (uint32_t)__half_as_ushort(__float2half_rn(sf)) * 0x00010001u;
                        const bool zero = (m24 & 0x7FFFu) == 0u;
                        m20 = zero ? 0u : m24 - 4u * 0x04000400u;
                        mc = zero ? 0u : (m24 - 21u * 0x04000400u) ^ 0x80008000u;
                    }
#pragma unroll
                    for (uint32_t c = 0; c < 2u; ++c) {
                        const uint4 p = *reinterpret_cast<const uint4*>(pk_row + ((c ? off1 : off0) ^ (jj * 64u)));
                        uint32_t m[2];     // multipliers of the chunk's first and second 16 columns
                        if (FMT == STRATA_MOE_FMT_MXFP4) {
                            // f16 exponent field e - emin + 2 in both halves (arithmetic modulo 2^32)
                            m[0] = m[1] = __byte_perm(sel[jj], 0u, 0x4440u + 2u * sub + c) * 0x04000400u + mx_add;
                        } else if (FMT == STRATA_MOE_FMT_NVFP4) {
                            uint32_t pair;
                            asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(pair) : "h"((unsigned short)(sel[jj] >> (16u * c))));
                            m[0] = __byte_perm(pair, pair, 0x1010);
                            m[1] = __byte_perm(pair, pair, 0x3232);
                        } else if (FMT == STRATA_MOE_FMT_INT4G128) {
                            const uint32_t h = __half_as_ushort(__float2half_rn(__uint_as_float(sel[jj] << 16)));
                            m[0] = m[1] = h * 0x00010001u;
                        }
                        const uint32_t w[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
                        for (uint32_t i = 0; i < 4u; ++i) {
                            uint32_t r[4];
                            if (FMT == kFmtInt4N) {
                                p_int4x8_narrow(w[i], m24, m20, mc, &v[c * 16u + i * 4u]);
                                continue;
                            }
                            if (FMT == STRATA_MOE_FMT_INT4G128) p_int4x8_f16(w[i], r);
                            else p_e2m1x8_f16(w[i], r);
#pragma unroll
                            for (uint32_t e = 0; e < 4u; ++e) v[c * 16u + i * 4u + e] = p_mul_f16x2(r[e], m[i >> 1]);
                        }
                    }
                    keep32(v);     // decoded before the wait below
                    if (jj == 1u || q * 4u + 2u >= k_slabs) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&S.pk_empty[rp.i]);  // this warp is done reading the block
                    }
                    if (!mbar_wait_warp(&S.empty_a[ra.i], ra.ph ^ 1u, abort_flag)) { ok = false; break; }
                    tc_fence_after();   // the MMAs that read this stage have completed
                    tmem_st32(a_lane + ra.i * G::kAStageCols, v);
                    tmem_st_wait();
                    tc_fence_before();   // order the tensor-memory stores before the MMA issuer's reads
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&S.full_a[ra.i]);
                    ra.next(kSlabs == 1u ? 2u : 1u);
                }
                if (!ok) break;
                rp.next();
                if (hn) {
                    if (q == 0u) {
                        sbase = wt.scales[tn.g];
                        if (kEmin) emin_n = wt.emin[tn.g];
                    }
                    if (q + 2u == blocks || blocks == 1u) srow = sbase + (tn.m0 + arow + which * kSecond) * scale_row;
                    if (blocks == 1u) sc_next = load_scales(srow, 0);
                }
            }
            t = tn;
            have = hn;
            emin = emin_n;
        }
        if (!ok) { *abort_flag = 1; atomicOr(a.status, kStatusWaitTimeout); }
    } else {
        // ---------------------------------------------------------------- epilogue
        const uint32_t ew = warp - kFirstEpilogueWarp;
        const uint32_t lane_base = (warp & 3u) * 32u;
        Ring<kAccBufs> rc;
        bool ok = true, bad = false;
        TileInfo t, tn;
        bool have = tile_lookup(a, blockIdx.x, total, m_tiles, t, kTileFeat);
        for (uint32_t tile = blockIdx.x; ok && have; tile += gridDim.x) {
            const bool hn = tile_lookup(a, tile + gridDim.x, total, m_tiles, tn, kTileFeat);
            constexpr bool kNoPost = FMT == STRATA_MOE_FMT_INT4G128 || BF;
            float s0, s1 = 1.0f;
            if (GU) {
                s0 = kNoPost ? 1.0f : a.gate.post_scale[t.g];
                s1 = kNoPost ? 1.0f : a.up.post_scale[t.g];
            } else {
                s0 = s1 = kNoPost ? 1.0f : a.down.post_scale[t.g];
            }
            // One warp polls, the others sleep on a hardware barrier that also carries its verdict: all warps leave after the
            // same tile.  (The abort flag is no verdict: another role may raise it between two warps' reads, and those that
            // missed it would meet the next barrier alone.)
            if (epilogue_vote(ew == 0u && !mbar_wait(&S.acc_full[rc.i], rc.ph, abort_flag))) { ok = false; break; }
            tc_fence_after();
            const uint32_t feat = t.m0 + lane_base + lane;
            const uint32_t act_col = FMT == STRATA_MOE_FMT_INT4G128 || FMT == kFmtInt4N ? int4_slot(feat) : feat;   // the down tiles' column order
            const uint32_t taddr = tmem_base + rc.i * (2u * NT) + (lane_base << 16);
            const uint32_t lo_at = 16u << box_of(t.n);      // SPLIT: accumulator columns of the lo rows
            for (uint32_t c0 = (ew >> 2) * 16u; c0 < t.n; c0 += 16u * (kEpilogueWarps / 4u)) {
                uint32_t g[16], u[16];
                tmem_ld16(taddr + c0, g);
                if (DUAL) tmem_ld16(taddr + NT + c0, u);
                tmem_ld_wait();
                if (SPLIT) {
                    uint32_t l[16];
                    tmem_ld16(taddr + lo_at + c0, l);
                    tmem_ld_wait();
#pragma unroll
                    for (uint32_t j = 0; j < 16u; ++j) g[j] = __float_as_uint(__uint_as_float(g[j]) + __uint_as_float(l[j]));
                    if (DUAL) {
                        tmem_ld16(taddr + NT + lo_at + c0, l);
                        tmem_ld_wait();
#pragma unroll
                        for (uint32_t j = 0; j < 16u; ++j) u[j] = __float_as_uint(__uint_as_float(u[j]) + __uint_as_float(l[j]));
                    }
                }
#pragma unroll
                for (uint32_t j = 0; j < 16u; ++j) {
                    if (c0 + j >= t.n) break;
                    const size_t pos = (size_t)t.row0 + c0 + j;
                    const float rs = rowscale ? rowscale[pos] : 1.0f;   // undoes the pre-scale of the activation row
                    if (GU) {
                        const float gv = __uint_as_float(g[j]) * s0 * rs, uv = __uint_as_float(u[j]) * s1 * rs;
                        float v;
                        if (a.glu.kind == STRATA_MOE_ACT_SWIGLU) {
                            const float e = __expf(-fabsf(gv));
                            const float sig = gv >= 0.0f ? __fdividef(1.0f, 1.0f + e) : __fdividef(e, 1.0f + e);
                            v = gv * sig * uv;
                        } else {
                            v = glu_other(gv, uv, a.glu);
                        }
                        if (!(fabsf(v) <= (BF || a.act_f32 ? 3.0e38f : 65504.0f))) bad = true;
                        if (!BF && a.act_f32) {
                            a.act_f32[pos * R + feat] = v;
                        } else if (BF) {
                            const __nv_bfloat16 h = __float2bfloat16_rn(v);
                            static_cast<__nv_bfloat16*>(act_out_v)[pos * R + act_col] = h;
                            if (a.act_lo) static_cast<__nv_bfloat16*>(a.act_lo)[pos * R + act_col] = __float2bfloat16_rn(v - __bfloat162float(h));
                        } else {
                            const __half h = __float2half_rn(v);
                            static_cast<__half*>(act_out_v)[pos * R + act_col] = h;
                        }
                    } else {
                        const float v = __uint_as_float(g[j]) * s0 * rs;
                        const float lim = a.y_half ? 65504.0f : 3.0e38f;
                        if (a.y_rowscale_out != nullptr && feat == 0u) a.y_rowscale_out[pos] = 1.0f;
                        if (!(fabsf(v) <= lim)) bad = true;
                        if (a.y_half) reinterpret_cast<__half*>(a.y)[pos * R + feat] = __float2half_rn(v);
                        else a.y[pos * R + feat] = v;
                        if (MODE == 2) {
                            const float v2 = __uint_as_float(u[j]) * s1 * rs;
                            if (!(fabsf(v2) <= lim)) bad = true;
                            if (a.y_half) reinterpret_cast<__half*>(a.y)[pos * R + feat + kMTile] = __float2half_rn(v2);
                            else a.y[pos * R + feat + kMTile] = v2;
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.acc_empty[rc.i]);
            rc.next();
            t = tn;
            have = hn;
        }
        if (!ok) { *abort_flag = 1; atomicOr(a.status, kStatusWaitTimeout); }
        if (bad) atomicOr(a.status, kStatusNonFiniteOutput);
    }

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// ------------------------------------------------------------------------------ tile list
// table[0] = number of n-tiles, then (expert, first row, rows) per n-tile, experts ascending.
__global__ void __launch_bounds__(1024) prefill_tiles_kernel(const uint32_t* offsets, uint32_t n_groups, uint32_t* table,
                                                             uint32_t kNTile) {
    __shared__ uint32_t scan[1024];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t tid = threadIdx.x;
    uint32_t cnt = 0, r0 = 0;
    if (tid < n_groups) {
        r0 = offsets[tid];
        cnt = offsets[tid + 1] - r0;
    }
    const uint32_t mine = (cnt + kNTile - 1) / kNTile;
    scan[tid] = mine;
    __syncthreads();
    for (uint32_t off = 1; off < 1024u; off <<= 1) {
        const uint32_t v = tid >= off ? scan[tid - off] : 0u;
        __syncthreads();
        scan[tid] += v;
        __syncthreads();
    }
    const uint32_t base = scan[tid] - mine;
    for (uint32_t i = 0; i < mine; ++i) {
        table[4 + 3 * (base + i)] = tid;
        table[4 + 3 * (base + i) + 1] = r0 + i * kNTile;
        table[4 + 3 * (base + i) + 2] = min(kNTile, cnt - i * kNTile);
    }
    if (tid == 1023u) table[0] = scan[1023];
}

// ------------------------------------------------------------------------------ host side
TensorMapEncodeFn tensor_map_encoder() {
    static TensorMapEncodeFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<TensorMapEncodeFn>(p);
    }
    return fn;
}

// 16-bit matrix [rows, cols] row-major; box = 64 columns x box_rows rows, 128-byte swizzle.
static bool make_map(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows) {
    TensorMapEncodeFn fn = tensor_map_encoder();
    if (!fn) return false;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};
    const cuuint32_t box[2] = {kBK, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool prefill_supported(int fmt, uint32_t H, uint32_t I) {
    if (fmt < 0 || fmt > kFmtBf16W) return false;
    return H % 128u == 0 && I % 128u == 0 && tensor_map_encoder() != nullptr;
}

size_t prefill_scratch_bytes(uint32_t n_groups, uint32_t pairs) {
    return (4 + 3 * ((size_t)pairs / kMinTileRows + n_groups + 1)) * sizeof(uint32_t);
}

static bool make_bmaps(BMaps* b, const void* base, uint64_t rows, uint64_t cols) {
    for (int i = 0; i < 4; ++i)
        if (!make_map(&b->m[i], base, rows, cols, 16u << i)) return false;
    return true;
}

// Tensor map over one projection's packed 4-bit rows ([rows, K/2] bytes): 128-byte x 128-row
// boxes, 128-byte swizzle.  `out` receives the 128-byte descriptor (host memory).
int prefill_encode_weight_map(void* out, const void* packed, uint32_t rows, uint32_t K) {
    TensorMapEncodeFn fn = tensor_map_encoder();
    if (!fn) return -1;
    const cuuint64_t dims[2] = {K / 2u, rows};
    const cuuint64_t strides[1] = {K / 2u};
    const cuuint32_t box[2] = {kPkCols / 2u, kMTile};
    const cuuint32_t estr[2] = {1, 1};
    static_assert(sizeof(CUtensorMap) == 128, "descriptor size");
    return fn(static_cast<CUtensorMap*>(out), CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(packed), dims,
              strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
               ? 0
               : -1;
}

// Alignment of a projection's scales that load_scales relies on: one load per 256-column block of a row when rows are
// whole blocks, the narrower loads otherwise.
uint32_t prefill_scale_align(int fmt, uint32_t K) {
    const bool whole_blocks = K % kPkCols == 0u;
    switch (fmt) {
        case STRATA_MOE_FMT_MXFP4: return whole_blocks ? 8u : 4u;
        case STRATA_MOE_FMT_NVFP4: return whole_blocks ? 16u : 8u;
        case STRATA_MOE_FMT_INT4G128: return whole_blocks ? 4u : 2u;
        default: return 1u;
    }
}

// Tensor map over one projection's BF16 rows ([rows, K]): boxes of 64 columns x 128 rows.
int prefill_encode_weight_map_bf16(void* out, const void* w, uint32_t rows, uint32_t K) {
    return make_map(static_cast<CUtensorMap*>(out), w, rows, K, kMTile) ? 0 : -1;
}

// One kernel launch.  b_hi / b_lo: the 16-bit activation rows [rows_cap, K] (b_lo only when SPLIT); map_a0 / map_a1: the
// weight matrices of a launch without a map table (wmaps == nullptr, BF16 only).
template <int FMT, int MODE, int NT, bool SPLIT>
static int launch_one(const PrefillArgs& a, const void* b_hi, const void* b_lo, uint32_t rows_cap,
                      const CUtensorMap* map_a0, const CUtensorMap* map_a1, const float* rowscale, void* act_out,
                      const void* wmaps, cudaStream_t s) {
    // the opt-in to more than 48 KB of dynamic shared memory is a per-device property of the function
    static bool done[64] = {};
    const size_t smem = sizeof(PrefillSmem<NT>) + 1024;
    static_assert(sizeof(PrefillSmem<NT>) + 1024 <= 227u * 1024u, "shared memory");
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -2;
    if (!done[dev]) {
        if (cudaFuncSetAttribute(prefill_ffn_kernel<FMT, MODE, NT, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem) != cudaSuccess)
            return -2;
        done[dev] = true;
    }
    BMaps hi, lo;
    const uint32_t K = MODE == 0 ? a.H : a.I;
    if (!make_bmaps(&hi, b_hi, rows_cap, K)) return -1;
    if (SPLIT) {
        if (!make_bmaps(&lo, b_lo, rows_cap, K)) return -1;
    } else {
        lo = hi;
    }
    prefill_ffn_kernel<FMT, MODE, NT, SPLIT><<<kNumSMs, kThreads, smem, s>>>(
        hi, lo, map_a0 ? *map_a0 : hi.m[0], map_a1 ? *map_a1 : hi.m[0], a, rowscale, act_out,
        static_cast<const CUtensorMap*>(wmaps));
    ++g_kernel_launches;
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int launch_tile_list(const uint32_t* offsets, uint32_t n_groups, uint32_t* table, uint32_t rows, cudaStream_t s) {
    if (rows < kMinTileRows) return -1;      // more tiles than the list has room for
    const cudaError_t e = launch_behind(prefill_tiles_kernel, 1, 1024, 0, s, offsets, n_groups, table, rows);
    ++g_kernel_launches;
    return e == cudaSuccess ? 0 : -3;
}
static int launch_tiles(const PrefillArgs& a, cudaStream_t s) { return launch_tile_list(a.offsets, a.n_groups, a.tile_table, a.ntile, s); }

// Operands of the gate/up or the down launch beside PrefillArgs.
struct Operands {
    const void *hi, *lo;
    uint32_t rows_cap;
    const CUtensorMap *a0, *a1;
    const float* rowscale;
    void* act_out;
    const void* wmaps;
};

template <int FMT>
static int launch_gate_up_nt(const PrefillArgs& a, const Operands& o, cudaStream_t s) {
    if (a.ntile <= 32u) return launch_one<FMT, 0, 32, false>(a, o.hi, nullptr, o.rows_cap, o.a0, o.a1, o.rowscale, o.act_out, o.wmaps, s);
    if (a.ntile <= 64u) return launch_one<FMT, 0, 64, false>(a, o.hi, nullptr, o.rows_cap, o.a0, o.a1, o.rowscale, o.act_out, o.wmaps, s);
    if (a.ntile <= 128u) return launch_one<FMT, 0, 128, false>(a, o.hi, nullptr, o.rows_cap, o.a0, o.a1, o.rowscale, o.act_out, o.wmaps, s);
    if (a.ntile <= 160u) return launch_one<FMT, 0, 160, false>(a, o.hi, nullptr, o.rows_cap, o.a0, o.a1, o.rowscale, o.act_out, o.wmaps, s);
    return launch_one<FMT, 0, 192, false>(a, o.hi, nullptr, o.rows_cap, o.a0, o.a1, o.rowscale, o.act_out, o.wmaps, s);
}
// o.lo set: the activation is a hi + lo pair and the tile holds twice the token rows.
template <int FMT>
static int launch_down_nt(const PrefillArgs& a, const Operands& o, cudaStream_t s) {
    if (o.lo) {
        if (a.H % 256u) return launch_one<FMT, 1, 128, true>(a, o.hi, o.lo, o.rows_cap, o.a0, o.a1, o.rowscale, nullptr, o.wmaps, s);
        if (a.ntile <= 16u) return launch_one<FMT, 2, 32, true>(a, o.hi, o.lo, o.rows_cap, o.a0, o.a1, o.rowscale, nullptr, o.wmaps, s);
        if (a.ntile <= 32u) return launch_one<FMT, 2, 64, true>(a, o.hi, o.lo, o.rows_cap, o.a0, o.a1, o.rowscale, nullptr, o.wmaps, s);
        return launch_one<FMT, 2, 128, true>(a, o.hi, o.lo, o.rows_cap, o.a0, o.a1, o.rowscale, nullptr, o.wmaps, s);
    }
    if (a.H % 256u) return launch_one<FMT, 1, 128, false>(a, o.hi, nullptr, o.rows_cap, o.a0, o.a1, o.rowscale, nullptr, o.wmaps, s);
    if (a.ntile <= 32u) return launch_one<FMT, 2, 32, false>(a, o.hi, nullptr, o.rows_cap, o.a0, o.a1, o.rowscale, nullptr, o.wmaps, s);
    if (a.ntile <= 64u) return launch_one<FMT, 2, 64, false>(a, o.hi, nullptr, o.rows_cap, o.a0, o.a1, o.rowscale, nullptr, o.wmaps, s);
    if (a.ntile <= 128u) return launch_one<FMT, 2, 128, false>(a, o.hi, nullptr, o.rows_cap, o.a0, o.a1, o.rowscale, nullptr, o.wmaps, s);
    if (a.ntile <= 160u) return launch_one<FMT, 2, 160, false>(a, o.hi, nullptr, o.rows_cap, o.a0, o.a1, o.rowscale, nullptr, o.wmaps, s);
    return launch_one<FMT, 2, 192, false>(a, o.hi, nullptr, o.rows_cap, o.a0, o.a1, o.rowscale, nullptr, o.wmaps, s);
}
static int gate_up_any(const PrefillArgs& a, const Operands& o, cudaStream_t s) {
    switch (a.fmt) {
        case STRATA_MOE_FMT_MXFP4: return launch_gate_up_nt<STRATA_MOE_FMT_MXFP4>(a, o, s);
        case STRATA_MOE_FMT_NVFP4: return launch_gate_up_nt<STRATA_MOE_FMT_NVFP4>(a, o, s);
        case STRATA_MOE_FMT_INT4G128:
            return a.narrow ? launch_gate_up_nt<kFmtInt4N>(a, o, s) : launch_gate_up_nt<STRATA_MOE_FMT_INT4G128>(a, o, s);
        case kFmtBf16W: return launch_gate_up_nt<kFmtBf16W>(a, o, s);
        default: return -1;
    }
}
static int down_any(const PrefillArgs& a, const Operands& o, cudaStream_t s) {
    switch (a.fmt) {
        case STRATA_MOE_FMT_MXFP4: return launch_down_nt<STRATA_MOE_FMT_MXFP4>(a, o, s);
        case STRATA_MOE_FMT_NVFP4: return launch_down_nt<STRATA_MOE_FMT_NVFP4>(a, o, s);
        case STRATA_MOE_FMT_INT4G128:
            return a.narrow ? launch_down_nt<kFmtInt4N>(a, o, s) : launch_down_nt<STRATA_MOE_FMT_INT4G128>(a, o, s);
        case kFmtBf16W: return launch_down_nt<kFmtBf16W>(a, o, s);
        default: return -1;
    }
}
// Tiles of shapes whose down projection takes single weight tiles (H % 256 == 128) hold at most 128 rows, or 64 pairs; none
// is smaller than the tile list has room for.
static PrefillArgs with_tile(PrefillArgs a, bool split) {
    const uint32_t most = split ? 64u : (a.H % 256u ? 128u : 192u);
    if (a.ntile != 0u && a.ntile < kMinTileRows) a.ntile = kMinTileRows;
    if (a.ntile == 0u || a.ntile > most) a.ntile = most;
    return a;
}

int launch_prefill_gate_up(const PrefillArgs& args, const void* x16, const float* x_rowscale, void* act16,
                           uint32_t pairs_cap, const void* wmaps, cudaStream_t s) {
    const PrefillArgs a = with_tile(args, args.act_lo != nullptr);
    if (const int rc = launch_tiles(a, s)) return rc;
    return gate_up_any(a, Operands{x16, nullptr, pairs_cap, nullptr, nullptr, x_rowscale, act16, wmaps}, s);
}

int launch_prefill_down(const PrefillArgs& args, const void* act16, const float* act_rowscale, uint32_t pairs_cap,
                        const void* wmaps, cudaStream_t s) {
    const PrefillArgs a = with_tile(args, args.act_lo != nullptr);
    if (!a.reuse_tiles)
        if (const int rc = launch_tiles(a, s)) return rc;
    return down_any(a, Operands{act16, a.act_lo, pairs_cap, nullptr, nullptr, act_rowscale, nullptr, wmaps}, s);
}

int launch_prefill(const PrefillArgs& args, const void* x16, const float* x_rowscale, void* act16,
                   uint32_t pairs_cap, const void* wmaps, cudaStream_t s, cudaEvent_t mid) {
    PrefillArgs a = args;
    const int rc = launch_prefill_gate_up(a, x16, x_rowscale, act16, pairs_cap, wmaps, s);
    if (rc) return rc;
    if (mid) cudaEventRecord(mid, s);
    a.reuse_tiles = 1;
    return launch_prefill_down(a, act16, nullptr, pairs_cap, wmaps, s);
}

// BF16 expert (the shared expert) over `rows` token rows in natural order: x [rows, H] BF16,
// gate/up [I, H], down [H, I] BF16, act (and args.act_lo: a hi + lo pair) [rows_cap, I] BF16 scratch, y [rows, H] fp32.
int launch_prefill_bf16(const PrefillArgs& args, const void* x, uint32_t rows, const void* w_gate, const void* w_up,
                        const void* w_down, void* act, uint32_t rows_cap, cudaStream_t s) {
    PrefillArgs a = with_tile(args, args.act_lo != nullptr);
    a.tile_table = nullptr;
    a.pairs = rows;
    CUtensorMap map_g, map_u, map_d;
    if (!make_map(&map_g, w_gate, a.I, a.H, kMTile) || !make_map(&map_u, w_up, a.I, a.H, kMTile) ||
        !make_map(&map_d, w_down, a.H, a.I, kMTile))
        return -1;
    const int rc = launch_gate_up_nt<kFmtBf16W>(a, Operands{x, nullptr, rows, &map_g, &map_u, nullptr, act, nullptr}, s);
    if (rc) return rc;
    return launch_down_nt<kFmtBf16W>(a, Operands{act, a.act_lo, rows_cap, &map_d, &map_d, nullptr, nullptr, nullptr}, s);
}

// Router projection on the tensor cores: logits[t, e] = sum_h x[t, h] * wg[e, h] for BF16 operands,
// FP32 accumulation in tensor memory.  The expert rows play the 128-feature M tiles and the tokens the
// N tiles of the single-GEMM modes (one group holding all T rows), so the output lands as [T, E] fp32.
// The summation order differs from the canonical lane-strided order: these logits feed the fast
// router, which re-derives everything that reaches the caller in the canonical order.
// Needs E % 128 == 0 and H % 128 == 0.
int launch_router_tc(const void* x, uint32_t T, const void* wg, uint32_t E, uint32_t H, float* logits, uint32_t* status,
                     cudaStream_t s) {
    if (E % 128u || H % 128u || T == 0u) return -1;
    CUtensorMap map_w;
    if (!make_map(&map_w, wg, E, H, kMTile)) return -1;
    PrefillArgs a{};
    a.fmt = kFmtBf16W;
    a.H = E;     // features of the single-GEMM modes
    a.I = H;     // their K
    a.n_groups = 1;
    a.pairs = T;
    a.y = logits;
    a.status = status;
    a.glu = GluParams{STRATA_MOE_ACT_SWIGLU, 1.0f, 1.0f};
    a.ntile = 128u;   // more tiles than the 192-token geometry gives, and a tile is short (E features x H)
    // 256 experts per job while that still gives every other SM a job; with few tokens (a rank's share of an
    // expert-parallel step) 128 per job: twice the jobs, each half as long (2048 tokens: 16 jobs otherwise)
    const uint64_t jobs256 = (uint64_t)((T + 127u) / 128u) * (E / 256u);
    if (E % 256u == 0u && jobs256 * 2u >= (uint64_t)kNumSMs)
        return launch_one<kFmtBf16W, 2, 128, false>(a, x, nullptr, T, &map_w, &map_w, nullptr, nullptr, nullptr, s);
    return launch_one<kFmtBf16W, 1, 128, false>(a, x, nullptr, T, &map_w, &map_w, nullptr, nullptr, nullptr, s);
}

}  // namespace smoe
