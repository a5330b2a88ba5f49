// Expert FFN of small groups for the FP4 formats on the block-scaled tensor-core instructions: no weight is decoded.
//
// tcgen05.mma kind::mxf4 / kind::mxf4nvf4 multiplies packed E2M1 values whose block scales (E8M0 per 32 columns, E4M3 per
// 16) are applied inside the instruction, which is MXFP4 and NVFP4 as they lie in the checkpoint.  The activations have to
// be E2M1 too; 24 bits of them travel as eight DIGIT PLANES: a block of a row (32 or 16 columns) is written in fixed point
// against the power of two below its largest value,
//     x = 2^b * sum over t of d_t * 8^-t,   d_t an E2M1 number, |d_t| <= 4,   |error| <= 2^(b - 22), mostly 2^(b - 23),
// that is at most 2^-23 of the block's maximum; BF16 values down to 2^-15 of it are exact.  A token row is thus eight
// rows of the N operand with one common set of block scales 2^b, and the epilogue adds the eight accumulators with the
// factors 8^-t.  The products are exact, the sums are the tensor core's FP32 accumulation.  A row with outliers in a block (see
// planes_kernel) comes with a second row of planes, the remainder that its digits leave; the epilogue adds it.
//
// Measured (gate/up of 4096 x 2048 x 256 MXFP4 experts, L2 flushed): 256 tokens 360 us, 6.3 TB/s; 8 tokens 77 us, 5.0 TB/s, the
// last round of tiles and the ramp being the rest.  The kernels that decode: ring 82 us at 8 tokens, tiles 3.5 TB/s.
//
// What bounds it: HBM, the packed weights, read once.  An M = 128, N = 8 rows, K = 64 instruction takes N / 2 clocks for
// 4 KB of weights, which HBM delivers to an SM in 178 clocks: up to 24 rows (N = 192) the tensor pipe keeps up, and a
// second pass over a larger group's weights still costs less than the decode that the f16 tiles pay.
//
//   warp 0        producer: packed weights (two TMA boxes of 128 rows x 256 columns per stage), the token rows (one bulk copy:
//                 a row's eight planes of 256 columns are exactly one 128-byte-swizzle atom, which the conversion lays out as
//                 the MMA reads it, rows of a group side by side), block scales (16 bytes per weight row and per token row)
//   warp 1        MMA issuer: one elected lane
//   warps 2..5    block scales: shared memory -> tensor memory (a scale is read by the MMA from the tensor-memory column
//                 of its row modulo 32, in all four lane quarters)
//   warps 6..13   epilogue: tcgen05.ld, sum of the planes, SwiGLU (gate/up), store
//
// Rows, not row tiles, are the unit of the N operand: a group of n rows, their remainders counted, costs N = 8 n (rounded to
// 16) columns.  CTAs are persistent and walk (group, row tile, 128 features of gate and up, or 256 of down) jobs, each in one
// pass over the weights, or more where the rows and their remainders are more than a tile holds.
//
// Every wait is bounded: on expiry the kernel raises kStatusWaitTimeout, all roles leave their loops, tensor memory is
// released and the kernel returns normally.
//
// Replaces the reference's per-row NVFP4 / DeepSeek FP4 expert kernels (kernels/cuda/backend.cu:1978-2069, 2308-2413).
#include <cuda.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "tc5.cuh"

namespace smoe {

namespace {

constexpr uint32_t kMT = 128;                    // weight rows per MMA
constexpr uint32_t kStageK = 256;                // columns per stage: 128 packed bytes of a weight row
constexpr uint32_t kWTile = kMT * (kStageK / 2u);
constexpr uint32_t kPlanes = 8;
constexpr uint32_t kRowBytes = kPlanes * (kStageK / 2u);   // one token row of a stage
constexpr uint32_t kSfTile = kMT * 16u;          // scales of 128 weight rows, 16 bytes each: 512 columns MXFP4, 256 NVFP4
constexpr uint32_t kSfStages = 4;
constexpr uint32_t kMaxCols = 8192;
constexpr uint32_t kSfBufs = 2;                  // scale buffers in tensor memory
constexpr uint32_t kEpiWarp0 = 6, kEpiWarps = 8;
constexpr uint32_t kPThreads = (kEpiWarp0 + kEpiWarps) * 32;

// R: most token rows per tile.
template <int R>
struct PGeo {
    static_assert(R == 8 || R == 16 || R == 24, "tile sizes");
    static constexpr uint32_t kN = kPlanes * R;
    static constexpr uint32_t kStages = R == 8 ? 5u : R == 16 ? 4u : 3u;
    static constexpr uint32_t kAccBufs = R == 8 ? 2u : 1u;
    static constexpr uint32_t kAccCols = kAccBufs * 2u * kN;
    static constexpr uint32_t kBGroups = R / 4u;                    // groups of 32 N rows = 4 token rows
    static constexpr uint32_t kBPitch = R <= 16 ? 4u : 8u;          // tensor-memory columns per scale word of the N operand
    static constexpr uint32_t kSfCols = 32u + 4u * kBPitch;         // four words of: weight tile 0, weight tile 1, rows
    static_assert(kAccCols + kSfBufs * kSfCols <= 512u, "tensor memory");
};

template <int R>
struct __align__(1024) PSmem {
    uint8_t w[PGeo<R>::kStages][2][kWTile];
    uint8_t b[PGeo<R>::kStages][R * kRowBytes];
    uint8_t sf[kSfStages][2][kSfTile];
    uint8_t sfb[kSfStages][R * 16u];                        // the token rows' block scales of the same columns
    uint64_t full[PGeo<R>::kStages], empty[PGeo<R>::kStages];
    uint64_t sfs_full[kSfStages], sfs_empty[kSfStages];     // scales in shared memory
    uint64_t sft_full[kSfBufs], sft_empty[kSfBufs];         // scales in tensor memory
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    uint32_t abort_flag;
};

// Instruction descriptor of kind::mxf4 / mxf4nvf4: E2M1 x E2M1, K-major, M = 128; scale type E8M0 or E4M3; sf_id: first
// scale byte of a 32-bit word that the instruction uses.
__device__ __forceinline__ uint32_t idesc_fp4(uint32_t n, bool e8m0, uint32_t sf_id) {
    return (sf_id << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((e8m0 ? 1u : 0u) << 23) | ((kMT >> 7) << 27) | (sf_id << 29);
}
// The four K = 64 MMAs of one 128-byte-swizzled stage of one weight tile.  sfa / sfb: scale words of the first; sfb_step: tensor-
// memory columns between the words of the rows' scales.  The branches on `never` (0, but not for the compiler) end the basic
// blocks: MMAs in straight-line code run without overlap (see umma4_f16_ts in prefill.cu).
template <bool MX>
__device__ __forceinline__ void mma4_fp4(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t id0, uint32_t id2, uint32_t sfa, uint32_t sfb,
                                         uint32_t sfb_step, uint32_t accumulate, uint32_t never) {
#define SMOE_MMA4(KIND, I1, I3, A1, A2, A3, B1, B2, B3)                                                                        \
    asm volatile(                                                                                                              \
        "{\n .reg .pred p, t, q;\n .reg .b64 a0, a1, a2, a3, b0, b1, b2, b3;\n .reg .b32 k1, k2, k3, l1, l2, l3;\n"             \
        " setp.ne.b32 p, %5, 0;\n setp.eq.b32 t, 0, 0;\n setp.ne.b32 q, %6, 0;\n"                                              \
        " add.u32 k1, %1, 2;\n add.u32 k2, %1, 4;\n add.u32 k3, %1, 6;\n add.u32 l1, %2, 2;\n add.u32 l2, %2, 4;\n"            \
        " add.u32 l3, %2, 6;\n mov.b64 a0, {%1, %7};\n mov.b64 a1, {k1, %7};\n mov.b64 a2, {k2, %7};\n mov.b64 a3, {k3, %7};\n" \
        " mov.b64 b0, {%2, %7};\n mov.b64 b1, {l1, %7};\n mov.b64 b2, {l2, %7};\n mov.b64 b3, {l3, %7};\n"                      \
        " tcgen05.mma.cta_group::1." KIND " [%0], a0, b0, %3, [%8], [%11], p;\n @q bra DONE;\n"                                \
        " tcgen05.mma.cta_group::1." KIND " [%0], a1, b1, " I1 ", [" A1 "], [" B1 "], t;\n @q bra DONE;\n"                     \
        " tcgen05.mma.cta_group::1." KIND " [%0], a2, b2, %3, [" A2 "], [" B2 "], t;\n @q bra DONE;\n"                         \
        " tcgen05.mma.cta_group::1." KIND " [%0], a3, b3, " I3 ", [" A3 "], [" B3 "], t;\n DONE:\n}" ::"r"(d),                 \
        "r"(a_lo), "r"(b_lo), "r"(id0), "r"(id2), "r"(accumulate), "r"(never), "n"(kDescHi), "r"(sfa), "r"(sfa + 4u),          \
        "r"(sfa + 8u), "r"(sfb), "r"(sfb + sfb_step), "r"(sfb + 2u * sfb_step), "r"(sfa + 12u), "r"(sfb + 3u * sfb_step)       \
        : "memory")
    // MXFP4: two scale bytes per MMA, the instruction descriptor says which half of the word; NVFP4: a word per MMA
    if (MX) SMOE_MMA4("kind::mxf4.block_scale.scale_vec::2X", "%4", "%4", "%8", "%9", "%9", "%11", "%12", "%12");
    else SMOE_MMA4("kind::mxf4nvf4.block_scale.scale_vec::4X", "%3", "%3", "%9", "%10", "%14", "%12", "%13", "%15");
#undef SMOE_MMA4
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t v[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
        "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t v[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}
// sum over t of v[t] * 8^-t, smallest terms first
__device__ __forceinline__ float plane_sum(const uint32_t v[8]) {
    float s = __uint_as_float(v[7]);
#pragma unroll
    for (int t = 6; t >= 0; --t) s = fmaf(s, 0.125f, __uint_as_float(v[t]));
    return s;
}

struct Job {
    uint32_t g, row0, n, m0;   // group, first row, rows (1 .. R), first output feature
};
// Job `job` of the launch: from the tile list, or (every group fits one tile) from the list of groups with rows.
__device__ __forceinline__ bool job_lookup(const PlaneArgs& a, uint32_t job, uint32_t total, uint32_t m_tiles, uint32_t feat, Job& j) {
    if (job >= total) return false;
    const uint32_t q = job / m_tiles;
    if (a.tile_table) {
        j.g = a.tile_table[4 + 3 * q];
        j.row0 = a.tile_table[4 + 3 * q + 1];
        j.n = a.tile_table[4 + 3 * q + 2];
    } else {
        j.g = a.active_list[q];
        j.row0 = a.offsets[j.g];
        j.n = min(a.offsets[j.g + 1] - j.row0, a.tile_rows);
    }
    j.m0 = (job - q * m_tiles) * feat;
    return true;
}
// A warp's way through its CTA's jobs.  The entry of the next job and, when that is there (`early`, half a pass later), the
// remainder factors of its rows are requested before they are needed.
template <bool REST>
struct Walk {
    const PlaneArgs& a;
    const uint32_t total, m_tiles, feat, lane;
    uint32_t job;
    bool have, have_next = false;
    Job j, next;
    float rest = 0.0f, rest_next = 0.0f;     // lane r: of row r
    uint32_t mask = 0;                       // rows that have a remainder
    __device__ __forceinline__ Walk(const PlaneArgs& args, uint32_t total_, uint32_t m_tiles_, uint32_t feat_, uint32_t lane_)
        : a(args), total(total_), m_tiles(m_tiles_), feat(feat_), lane(lane_), job(blockIdx.x) {
        have = job_lookup(a, job, total, m_tiles, feat, j);
        if (REST && have) take(lane < j.n ? a.x.rest_factor[j.row0 + lane] : 0.0f);
    }
    __device__ __forceinline__ void take(float r) {
        rest = r;
        mask = __ballot_sync(0xFFFFFFFFu, r != 0.0f);
    }
    __device__ __forceinline__ void look_ahead() { have_next = job_lookup(a, job + gridDim.x, total, m_tiles, feat, next); }
    __device__ __forceinline__ void early() {
        if (REST) rest_next = have_next && lane < next.n ? a.x.rest_factor[next.row0 + lane] : 0.0f;
    }
    __device__ __forceinline__ void advance() {
        job += gridDim.x;
        have = have_next;
        j = next;
        if (REST) take(rest_next);
    }
};
// One pass over the job's weights: the rows r0 .. r0 + rows - 1, as many as fit R rows together with their remainders, which
// follow them in the N operand.
struct Pass {
    uint32_t rows, part;      // part: those of them that have a remainder, bit i = row r0 + i
    __device__ __forceinline__ uint32_t count() const { return rows + __popc(part); }
};
template <int R, bool REST>
__device__ __forceinline__ Pass pass_from(const Walk<REST>& w, uint32_t r0) {
    if (!REST) return Pass{w.j.n, 0u};
    const uint32_t rest = w.mask >> r0;
    const bool fits = r0 + w.lane < w.j.n && w.lane + 1u + __popc(rest & ((2u << w.lane) - 1u)) <= (uint32_t)R;
    const uint32_t rows = __popc(__ballot_sync(0xFFFFFFFFu, fits));
    return Pass{rows, rest & ((1u << rows) - 1u)};
}

// GU: gate and up tiles of the same 128 features, SwiGLU, act (FP32) out, K = H.  Else two adjacent down tiles (256 features),
// y (FP32) out, K = I.
// REST: some row of the launch has a remainder.  The roles of the CTA until no jobs are left or a wait ran out (false).
template <int FMT, bool GU, int R, bool REST>
__device__ __forceinline__ bool plane_roles(const PlaneArgs& a, const CUtensorMap* wmaps, const CUtensorMap* smaps, PSmem<R>& S, uint32_t tm,
                                            uint32_t total) {
    using G = PGeo<R>;
    constexpr bool MX = FMT == STRATA_MOE_FMT_MXFP4;
    constexpr uint32_t kPerSf = MX ? 2u : 1u;      // stages per 16 scale bytes
    constexpr uint32_t kFeat = GU ? kMT : 2u * kMT, kSecond = GU ? 0u : kMT;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t K = GU ? a.H : a.I, rows_out = GU ? a.I : a.H;
    const uint32_t m_tiles = rows_out / kFeat, k_stages = K / kStageK, sf_blocks = k_stages / kPerSf;
    volatile uint32_t* abort_flag = &S.abort_flag;
    bool ok = true;
    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        uint32_t issued = 0, sf_issued = 0;
        Ring<G::kStages> rb;
        Ring<kSfStages> rs;
        Walk<REST> w(a, total, m_tiles, kFeat, lane);
        for (; ok && w.have; w.advance()) {
            w.look_ahead();
            const Job& j = w.j;
            const size_t at0 = (size_t)(GU ? 0u : 2u) * a.n_groups + j.g, at1 = (size_t)(GU ? 1u : 2u) * a.n_groups + j.g;
            for (uint32_t r0 = 0; ok && r0 < j.n;) {
                const Pass p = pass_from<R>(w, r0);
                const uint32_t row = j.row0 + r0, count = p.count();
                const bool rest = (p.part >> lane) & 1u;      // this lane fetches the remainder of row `row + lane`
                const uint32_t rest_at = p.rows + __popc(p.part & ((1u << lane) - 1u));
                for (uint32_t ks = 0; ks < k_stages; ++ks) {
                    // few large requests: one per token row and stage (24 + 2) took longer to issue than the weights to arrive (3072 x
                    // 1024 x 256 NVFP4 experts of 20 rows: gate/up 223 us); remainders, which few rows have, take one each
                    if (ks % kPerSf == 0u) {
                        const uint32_t blk = ks / kPerSf;
                        if (!mbar_wait_warp(&S.sfs_empty[rs.i], rs.ph ^ 1u, abort_flag)) { ok = false; break; }
                        if (lane == 0) mbar_arrive_expect_tx(&S.sfs_full[rs.i], 2u * kSfTile + count * 16u);
                        __syncwarp();
                        if (lane < 2u)
                            tma_load_2d(S.sf[rs.i][lane], smaps + (lane ? at1 : at0), blk * 16u, j.m0 + lane * kSecond, &S.sfs_full[rs.i]);
                        else if (lane == 2u)
                            bulk_load(S.sfb[rs.i], a.x.scales + ((size_t)blk * a.x.rows + row) * 16u, p.rows * 16u, &S.sfs_full[rs.i]);
                        if (REST && rest)
                            bulk_load(S.sfb[rs.i] + rest_at * 16u, a.x.rest_scales + ((size_t)blk * a.x.rows + row + lane) * 16u, 16u,
                                      &S.sfs_full[rs.i]);
                        ++sf_issued;
                        rs.next();
                    }
                    if (!mbar_wait_warp(&S.empty[rb.i], rb.ph ^ 1u, abort_flag)) { ok = false; break; }
                    if (lane == 0) mbar_arrive_expect_tx(&S.full[rb.i], 2u * kWTile + count * kRowBytes);
                    __syncwarp();
                    if (lane < 2u)
                        tma_load_2d(S.w[rb.i][lane], wmaps + (lane ? at1 : at0), ks * (kStageK / 2u), j.m0 + lane * kSecond, &S.full[rb.i]);
                    else if (lane == 2u)
                        bulk_load(S.b[rb.i], a.x.planes + ((size_t)ks * a.x.rows + row) * kRowBytes, p.rows * kRowBytes, &S.full[rb.i]);
                    if (REST && rest)
                        bulk_load(S.b[rb.i] + rest_at * kRowBytes, a.x.rest_planes + ((size_t)ks * a.x.rows + row + lane) * kRowBytes, kRowBytes,
                                  &S.full[rb.i]);
                    ++issued;
                    rb.next();
                    if (ks == k_stages / 2u) w.early();
                }
                r0 += p.rows;
            }
        }
        if (lane == 0) {
            if (!ok) *abort_flag = 1;
            if (*abort_flag) {
                drain_copies(S.full, issued, G::kStages);
                drain_copies(S.sfs_full, sf_issued, kSfStages);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        // the whole warp walks the loop with values the compiler can prove uniform, one elected lane issues
        auto uni = [](uint32_t v) { return __shfl_sync(0xFFFFFFFFu, v, 0); };
        const bool el = elect_one();
        const uint32_t tmu = uni(tm);
        const uint32_t a_lo0 = umma_desc_lo(smem_u32(S.w[0][0])), b_lo0 = umma_desc_lo(smem_u32(S.b[0]));
        Ring<G::kStages> rb;
        Ring<kSfBufs> rs;
        Ring<G::kAccBufs> rc;
        Walk<REST> w(a, uni(total), m_tiles, kFeat, lane);
        for (; ok && w.have; w.advance()) {
            w.look_ahead();
            const uint32_t rows = uni(w.j.n);
            for (uint32_t r0 = 0; ok && r0 < rows;) {
                const Pass p = pass_from<R>(w, r0);
                const uint32_t n = kPlanes * ((uni(p.count()) + 1u) & ~1u);
                if (!mbar_wait_warp(&S.acc_empty[rc.i], rc.ph ^ 1u, abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint32_t id0 = idesc_fp4(n, MX, 0u), id2 = idesc_fp4(n, MX, 2u);
                const uint32_t d = tmu + rc.i * (2u * G::kN);
                for (uint32_t ks = 0; ks < k_stages; ++ks) {
                    if (ks % kPerSf == 0u && !mbar_wait_warp(&S.sft_full[rs.i], rs.ph, abort_flag)) { ok = false; break; }
                    if (!mbar_wait_warp(&S.full[rb.i], rb.ph, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_lo = a_lo0 + rb.i * (2u * kWTile >> 4), b_lo = b_lo0 + rb.i * (R * kRowBytes >> 4);
                    const uint32_t half = MX ? (ks % kPerSf) * 2u : 0u;       // first scale word of the stage
                    const uint32_t sfa = tmu + G::kAccCols + rs.i * G::kSfCols + half * 4u;
                    const uint32_t sfb = tmu + G::kAccCols + rs.i * G::kSfCols + 32u + half * G::kBPitch;
                    if (el) {
                        mma4_fp4<MX>(d, a_lo, b_lo, id0, id2, sfa, sfb, G::kBPitch, ks, a.H == 0u);
                        mma4_fp4<MX>(d + G::kN, a_lo + (kWTile >> 4), b_lo, id0, id2, sfa + 16u, sfb, G::kBPitch, ks, a.H == 0u);
                        umma_commit(&S.empty[rb.i]);
                        if ((ks + 1u) % kPerSf == 0u) umma_commit(&S.sft_empty[rs.i]);
                        if (ks + 1u == k_stages) umma_commit(&S.acc_full[rc.i]);
                    }
                    __syncwarp();
                    rb.next();
                    if ((ks + 1u) % kPerSf == 0u) rs.next();
                    if (ks == k_stages / 2u) w.early();
                }
                rc.next();
                r0 += uni(p.rows);
            }
        }
        if (!ok && lane == 0) *abort_flag = 1;
    } else if (warp < kEpiWarp0) {
        // ------------------------------------------------------------------ block scales -> tensor memory
        const uint32_t lanes_at = tm + ((warp & 3u) * 32u << 16) + G::kAccCols;
        Ring<kSfStages> rs;
        Ring<kSfBufs> rt;
        Walk<REST> w(a, total, m_tiles, kFeat, lane);
        for (; ok && w.have; w.advance()) {
            w.look_ahead();
            for (uint32_t r0 = 0; ok && r0 < w.j.n; r0 += pass_from<R>(w, r0).rows) {
                for (uint32_t b = 0; b < sf_blocks; ++b) {
                    if (!mbar_wait_warp(&S.sfs_full[rs.i], rs.ph, abort_flag)) { ok = false; break; }
                    // N row 32 q + lane belongs to token row 4 q + lane / 8 (rows past the tile's keep what was there: their columns
                    // of the accumulators are not read)
                    uint32_t vb[4u * G::kBPitch];
#pragma unroll
                    for (uint32_t q = 0; q < G::kBPitch; ++q) {
                        const uint4 v = *reinterpret_cast<const uint4*>(S.sfb[rs.i] + ((q < G::kBGroups ? q : 0u) * 4u + (lane >> 3)) * 16u);
                        vb[q] = v.x;
                        vb[G::kBPitch + q] = v.y;
                        vb[2u * G::kBPitch + q] = v.z;
                        vb[3u * G::kBPitch + q] = v.w;
                    }
                    uint32_t va[2][16];
#pragma unroll
                    for (uint32_t m = 0; m < 2u; ++m)
#pragma unroll
                        for (uint32_t q = 0; q < 4u; ++q) {
                            const uint4 v = *reinterpret_cast<const uint4*>(S.sf[rs.i][m] + (32u * q + lane) * 16u);
                            va[m][q] = v.x;
                            va[m][4u + q] = v.y;
                            va[m][8u + q] = v.z;
                            va[m][12u + q] = v.w;
                        }
                    __syncwarp();
                    if (!mbar_wait_warp(&S.sft_empty[rt.i], rt.ph ^ 1u, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t at = lanes_at + rt.i * G::kSfCols;
                    tmem_st16(at, va[0]);
                    tmem_st16(at + 16u, va[1]);
                    if (G::kBPitch == 4u) tmem_st16(at + 32u, vb);
                    else tmem_st32(at + 32u, vb);
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&S.sfs_empty[rs.i]);
                        mbar_arrive(&S.sft_full[rt.i]);
                    }
                    rs.next();
                    rt.next();
                    if (b == sf_blocks / 2u) w.early();
                }
            }
        }
        if (!ok && lane == 0) *abort_flag = 1;
    } else {
        // ------------------------------------------------------------------ epilogue
        const uint32_t ew = warp - kEpiWarp0;
        const uint32_t lane_base = (warp & 3u) * 32u;
        Ring<G::kAccBufs> rc;
        bool bad = false;
        Walk<REST> w(a, total, m_tiles, kFeat, lane);
        for (; ok && w.have; w.advance()) {
            // what the tile needs from memory comes in before its accumulators are waited for: lane r holds row r's factors
            const Job& j = w.j;
            w.look_ahead();
            const float factor = a.x.factor && lane < j.n ? a.x.factor[j.row0 + lane] : 1.0f;
            const float s0 = a.post0 ? a.post0[j.g] : 1.0f, s1 = a.post1 ? a.post1[j.g] : 1.0f;
            w.early();
            const uint32_t feat = j.m0 + lane_base + lane;
            for (uint32_t r0 = 0; r0 < j.n;) {
                const Pass p = pass_from<R>(w, r0);
                if (group_vote<kEpiWarps * 32u>(ew == 0u && !mbar_wait(&S.acc_full[rc.i], rc.ph, abort_flag))) { ok = false; break; }
                tc_fence_after();
                const uint32_t taddr = tm + rc.i * (2u * G::kN) + (lane_base << 16);
                for (uint32_t i = ew >> 2; i < p.rows; i += 2u) {
                    uint32_t v0[8], v1[8];
                    tmem_ld8(taddr + i * kPlanes, v0);
                    tmem_ld8(taddr + G::kN + i * kPlanes, v1);
                    tmem_ld_wait();
                    const uint32_t pos = j.row0 + r0 + i;
                    const float rsc = __shfl_sync(0xFFFFFFFFu, factor, r0 + i);
                    float v = plane_sum(v0) * s0 * rsc, u = plane_sum(v1) * s1 * rsc;
                    if (REST && ((p.part >> i) & 1u)) {
                        const uint32_t at = taddr + (p.rows + __popc(p.part & ((1u << i) - 1u))) * kPlanes;
                        tmem_ld8(at, v0);
                        tmem_ld8(at + G::kN, v1);
                        tmem_ld_wait();
                        const float rest = __shfl_sync(0xFFFFFFFFu, w.rest, r0 + i);
                        v = fmaf(plane_sum(v0) * s0, rest, v);
                        u = fmaf(plane_sum(v1) * s1, rest, u);
                    }
                    if (GU) {
                        float o;
                        if (a.glu.kind == STRATA_MOE_ACT_SWIGLU) {
                            const float e = __expf(-fabsf(v));
                            const float sig = v >= 0.0f ? __fdividef(1.0f, 1.0f + e) : __fdividef(e, 1.0f + e);
                            o = v * sig * u;
                        } else {
                            o = glu_other(v, u, a.glu);
                        }
                        if (!(fabsf(o) <= 3.0e38f)) bad = true;
                        a.out[(size_t)pos * rows_out + feat] = o;
                    } else {
                        if (!(fabsf(v) <= 3.0e38f) || !(fabsf(u) <= 3.0e38f)) bad = true;
                        a.out[(size_t)pos * rows_out + feat] = v;
                        a.out[(size_t)pos * rows_out + feat + kMT] = u;
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&S.acc_empty[rc.i]);
                rc.next();
                r0 += p.rows;
            }
        }
        if (!ok) *abort_flag = 1;
        if (bad) atomicOr(a.status, kStatusNonFiniteOutput);
    }
    return ok;
}

// Registers: 80 a thread for the smallest tile leave an SM room for a CTA of the shared expert's streaming kernel beside this one
// and the activation's conversion, which is how a step of few tokens runs.  With the 90 that the remainders' loops ask for (the
// cap spills 6 bytes there) one of them waited: 1 token of 3072 x 1024 x 256 NVFP4 with the shared expert 63 - 78 us, capped 55, before
// the remainders 53; 4 tokens 84 - 103, 88, 84.  Larger tiles measured the same with and without.
template <int FMT, bool GU, int R>
__global__ void __maxnreg__(R == 8 ? 80 : 112)
fp4_planes_kernel(PlaneArgs a, const CUtensorMap* __restrict__ wmaps, const CUtensorMap* __restrict__ smaps /* both [3][n_groups] */) {
    using G = PGeo<R>;
    constexpr uint32_t kFeat = GU ? kMT : 2u * kMT;
    extern __shared__ uint8_t smem_raw_p[];
    PSmem<R>& S = *reinterpret_cast<PSmem<R>*>((reinterpret_cast<uintptr_t>(smem_raw_p) + 1023) & ~uintptr_t(1023));
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    pdl_launch_dependents();

    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < G::kStages; ++i) {
            mbar_init(&S.full[i], 1);
            mbar_init(&S.empty[i], 1);
        }
        for (uint32_t i = 0; i < kSfStages; ++i) {
            mbar_init(&S.sfs_full[i], 1);
            mbar_init(&S.sfs_empty[i], 4);
        }
        for (uint32_t i = 0; i < 2u; ++i) {
            mbar_init(&S.sft_full[i], 4);
            mbar_init(&S.sft_empty[i], 1);
            mbar_init(&S.acc_full[i], 1);
            mbar_init(&S.acc_empty[i], kEpiWarps);
        }
        S.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem_base)), "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = S.tmem_base;
    pdl_wait();      // what the roles read comes from the kernels before
    const uint32_t total = (a.tile_table ? a.tile_table[0] : *a.n_active) * ((GU ? a.I : a.H) / kFeat);
    // calls without outliers (nearly all) run the loops that know of no remainders
    const bool ok = *a.x.any_rest == a.x.call ? plane_roles<FMT, GU, R, true>(a, wmaps, smaps, S, tm, total)
                                              : plane_roles<FMT, GU, R, false>(a, wmaps, smaps, S, tm, total);
    if (!ok && lane == 0) atomicOr(a.status, kStatusWaitTimeout);

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm), "r"(512u) : "memory");
}

// ------------------------------------------------------------------------------ rows -> digit planes
// Eight columns of a thread, r = x * f1 with |r| <= 4 -> eight 32-bit words, word t = digit t of the columns (nibble c = column
// c).  A digit is the E2M1 number nearest to the rest, at most 1/2 away from it (1/4 below 2), and eight times what is left
// is the next rest; what the last digit leaves, times 8^8, stays in r.  All steps are exact in FP32.
__device__ __forceinline__ void digit_words(float r[8], uint32_t w[kPlanes]) {
#pragma unroll
    for (uint32_t t = 0; t < kPlanes; ++t) {
        uint32_t v[4];
        asm("{\n .reg .b8 b0, b1, b2, b3;\n"
            " cvt.rn.satfinite.e2m1x2.f32 b0, %6, %5;\n cvt.rn.satfinite.e2m1x2.f32 b1, %8, %7;\n"
            " cvt.rn.satfinite.e2m1x2.f32 b2, %10, %9;\n cvt.rn.satfinite.e2m1x2.f32 b3, %12, %11;\n"
            " mov.b32 %0, {b0, b1, b2, b3};\n"
            " cvt.rn.f16x2.e2m1x2 %1, b0;\n cvt.rn.f16x2.e2m1x2 %2, b1;\n"
            " cvt.rn.f16x2.e2m1x2 %3, b2;\n cvt.rn.f16x2.e2m1x2 %4, b3;\n}"
            : "=r"(w[t]), "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
            : "f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]));
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) {
            const float2 d = __half22float2(*reinterpret_cast<const __half2*>(&v[q]));
            r[2 * q] = (r[2 * q] - d.x) * 8.0f;
            r[2 * q + 1] = (r[2 * q + 1] - d.y) * 8.0f;
        }
    }
}
// The largest magnitude (as bits: exponent order is integer order, NaN and infinity come out on top) of a scale block, which
// four threads (MXFP4) or two hold.
template <int FMT>
__device__ __forceinline__ uint32_t block_max(const float x[8]) {
    uint32_t mx = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) mx = max(mx, __float_as_uint(x[c]) & 0x7FFFFFFFu);
    mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 1));
    if (FMT == STRATA_MOE_FMT_MXFP4) mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 2));
    return mx;
}
// 2^e as E4M3, e from -9 to 8
__device__ __forceinline__ uint32_t e4m3_pow2(int32_t e) { return e >= -6 ? (uint32_t)(e + 7) << 3 : 1u << (e + 9); }

// One CTA per source row (and, of a few rows, one per destination: blockIdx.y), eight columns per thread (cols <= 8192, a
// multiple of 256).  The row goes to the plane rows
// dest[row * k .. + k - 1] (0xFFFFFFFF: none), or to plane row `row`.
//   planes  [cols / 256][rows][8 planes][128 bytes], 16-byte chunk c of plane t at chunk c ^ t (the 128-byte swizzle)
//   scales  [cols / 512 (E8M0) or cols / 256 (E4M3)][rows][16]
// An E4M3 power of two spans 2^-9 .. 2^8: NVFP4 rows get a factor that puts their largest block at 2^8, and blocks more than
// 2^17 below it keep the smallest scale (an error of at most 2^-40 of the row's maximum).
//
// Rows with outliers: eight digits leave an error of 2^-23 of the block's maximum, which is nothing beside the block's own sum
// but much beside the rest of the block where an output's weights at the outliers are zero (4096 columns of N(0, 1) with one
// column 2^12, 2^16 or 2^20 times as large and a zero weight there: relative errors of 4e-6, 1.6e-4 and 4e-3).  A row gets a
// REMAINDER, what the digits leave written as a second row of digit planes with scales of its own (another 24 bits: an error
// of at most 2^-46 of the block's maximum), when in one of its blocks the digits are not exact and at least three quarters of
// the columns that are not zero lie 2^7 or more below the maximum.  In all other blocks the digits keep 2^-16 or better of more
// than a quarter of their columns.  N(0, 1) token rows never have one, the SwiGLU of N(0, 1.7^2) gates and ups in 2e-6 of its
// blocks of 16 and in none of 10^6 blocks of 32.
template <int FMT, bool F32>
__global__ void __launch_bounds__(1024) planes_kernel(const void* src, const uint32_t* rows_dev, uint32_t cols, const uint32_t* dest,
                                                      uint32_t k, PlaneRows o, bool settled) {
    __shared__ uint32_t warp_max[32];
    constexpr bool MX = FMT == STRATA_MOE_FMT_MXFP4;
    const uint32_t row = blockIdx.x, tid = threadIdx.x, lane = tid & 31u;
    pdl_launch_dependents();
    if (!settled) pdl_wait();
    if (rows_dev && row >= *rows_dev) return;
    float x[8];
    if (F32) {
        const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(src) + (size_t)row * cols) + 2u * tid;
        const float4 v0 = p[0], v1 = p[1];
        x[0] = v0.x; x[1] = v0.y; x[2] = v0.z; x[3] = v0.w; x[4] = v1.x; x[5] = v1.y; x[6] = v1.z; x[7] = v1.w;
    } else {
        const uint4 v = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(src) + (size_t)row * cols)[tid];
        const uint32_t h[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            x[2 * q] = __uint_as_float(h[q] << 16);
            x[2 * q + 1] = __uint_as_float(h[q] & 0xFFFF0000u);
        }
    }
    const uint32_t mx = block_max<FMT>(x);
    const uint32_t e = mx >> 23;      // biased exponent of the block's maximum
    constexpr uint32_t kPerScale = MX ? 4u : 2u;     // threads per block
    auto row_max = [&](uint32_t v) {
        const uint32_t wmax = __reduce_max_sync(0xFFFFFFFFu, v);
        if (lane == 0) warp_max[tid >> 5] = wmax;
        __syncthreads();
        return __reduce_max_sync(0xFFFFFFFFu, lane < blockDim.x / 32u ? warp_max[lane] : 0u);
    };
    uint32_t byte;
    float f1, row_factor = 1.0f;
    int32_t er = 0, sfe = 0;
    if (MX) {
        // block scale 2^(e - 128): the maximum lands in [2, 4)
        byte = e == 255u ? 255u : (e ? e - 1u : 0u);
        f1 = e == 255u ? 0.0f : __uint_as_float((254u - byte) << 23);
    } else {
        er = max((int32_t)(row_max(mx) >> 23), 20);
        sfe = max((int32_t)e - er + 8, -9);
        byte = e == 255u ? 0x7Fu : e4m3_pow2(sfe);
        f1 = e == 255u ? 0.0f : __uint_as_float((uint32_t)(136 - er - sfe + 127) << 23);
        row_factor = __uint_as_float((uint32_t)(er - 9) << 23);
    }
    float r[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) r[c] = e == 255u ? 0.0f : x[c] * f1;      // e = 255: the scale is NaN; the digits must not be
    uint32_t w[kPlanes];
    digit_words(r, w);
    // columns that are not zero | those far below the maximum << 8 | those that the digits do not hold exactly << 16
    uint32_t seen = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const uint32_t m = __float_as_uint(x[c]) & 0x7FFFFFFFu;
        seen += (m != 0u ? 1u : 0u) + (m != 0u && m + (7u << 23) <= mx ? 1u << 8 : 0u) + (r[c] != 0.0f ? 1u << 16 : 0u);
    }
    seen += __shfl_xor_sync(0xFFFFFFFFu, seen, 1);
    if (MX) seen += __shfl_xor_sync(0xFFFFFFFFu, seen, 2);
    if (settled) pdl_wait();     // the digits were made beside the preceding kernel; where they go it decides
    const uint32_t slab = tid >> 5, chunk = lane >> 2, word = lane & 3u, sc = tid / kPerScale;
    auto store = [&](uint8_t* planes, uint8_t* scales, uint32_t scale_byte, float* factor, float* rest_factor, float rest) {
        for (uint32_t j = blockIdx.y; j < (dest ? k : 1u); j += gridDim.y) {
            const uint32_t pos = dest ? dest[(size_t)row * k + j] : row;
            if (pos >= o.rows) continue;
            uint32_t* out = reinterpret_cast<uint32_t*>(planes + ((size_t)slab * o.rows + pos) * kRowBytes);
#pragma unroll
            for (uint32_t t = 0; t < kPlanes; ++t) out[t * 32u + ((chunk ^ t) << 2) + word] = w[t];
            if (tid % kPerScale == 0u) scales[((size_t)(sc >> 4) * o.rows + pos) * 16u + (sc & 15u)] = (uint8_t)scale_byte;
            if (tid == 0u) {
                if (factor) factor[pos] = row_factor;
                rest_factor[pos] = rest;
            }
        }
    };
    store(o.planes, o.scales, byte, MX ? nullptr : o.factor, o.rest_factor, 0.0f);
    if (!__syncthreads_or(seen >> 16 && 4u * ((seen >> 8) & 255u) >= 3u * (seen & 255u))) return;
    // the remainder: a unit of r is 2^-24 units of the digits' scale; the largest of a block lands in [2, 4) where the scales reach
    const uint32_t e2 = block_max<FMT>(r) >> 23;
    uint32_t byte2;
    int32_t f2;       // exponent of what r is multiplied by
    float rest_factor = 1.0f;
    if (MX) {
        byte2 = e2 ? (uint32_t)max((int32_t)byte + (int32_t)e2 - 152, 0) : 0u;
        f2 = (int32_t)byte - 24 - (int32_t)byte2;
    } else {
        const int32_t top = (int32_t)row_max(e2 ? (uint32_t)((int32_t)e2 + sfe + 16) : 0u) - 16;
        const int32_t sfe2 = e2 ? max((int32_t)e2 + sfe - top + 8, -9) : -9;
        byte2 = e4m3_pow2(sfe2);
        f2 = 136 + sfe - sfe2 - top;
        const int32_t at = top + er - 169;      // the factor's biased exponent
        rest_factor = __uint_as_float(at >= 1 ? (uint32_t)at << 23 : (at > -23 ? 1u << (22 + at) : 0u));
    }
    const float scale = e2 ? __uint_as_float((uint32_t)(f2 + 127) << 23) : 0.0f;
#pragma unroll
    for (int c = 0; c < 8; ++c) r[c] *= scale;
    digit_words(r, w);
    store(o.rest_planes, o.rest_scales, byte2, nullptr, o.rest_factor, rest_factor);
    if (tid == 0u) *o.any_rest = o.call;
}

template <int FMT, bool GU, int R>
int launch_planes_one(const PlaneArgs& a, const void* wmaps, const void* smaps, cudaStream_t s) {
    static bool done[64] = {};   // the shared-memory opt-in is per device
    const size_t smem = sizeof(PSmem<R>) + 1024;
    static_assert(sizeof(PSmem<R>) + 1024 <= 227u * 1024u, "shared memory");
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -2;
    if (!done[dev]) {
        if (cudaFuncSetAttribute(fp4_planes_kernel<FMT, GU, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
            return -2;
        done[dev] = true;
    }
    const cudaError_t e = launch_behind(fp4_planes_kernel<FMT, GU, R>, kNumSMs, kPThreads, smem, s, a,
                                        static_cast<const CUtensorMap*>(wmaps), static_cast<const CUtensorMap*>(smaps));
    ++g_kernel_launches;
    return e == cudaSuccess ? 0 : -3;
}
template <int FMT, bool GU>
int launch_planes_rows(const PlaneArgs& a, const void* wmaps, const void* smaps, cudaStream_t s) {
    switch (a.tile_rows) {      // a tile of more rows than the kernel's stages hold would be copied past their end
        case 8u: return launch_planes_one<FMT, GU, 8>(a, wmaps, smaps, s);
        case 16u: return launch_planes_one<FMT, GU, 16>(a, wmaps, smaps, s);
        case 24u: return launch_planes_one<FMT, GU, 24>(a, wmaps, smaps, s);
        default: return -1;
    }
}

template <int FMT>
void launch_planes_fmt(const void* src, bool f32, uint32_t rows, const uint32_t* rows_dev, uint32_t cols, const uint32_t* dest,
                       uint32_t k, const PlaneRows& out, bool settled, cudaStream_t s) {
    // the digits of a row are quickly made again: with few rows the copies of a row go to CTAs of their own
    const dim3 grid(rows, dest && rows * k <= 2u * (uint32_t)kNumSMs ? k : 1u);
    if (f32) launch_behind(planes_kernel<FMT, true>, grid, cols / 8u, 0, s, src, rows_dev, cols, dest, k, out, settled);
    else launch_behind(planes_kernel<FMT, false>, grid, cols / 8u, 0, s, src, rows_dev, cols, dest, k, out, settled);
}

}  // namespace

// A stage is 256 columns, a block of scales 16 bytes per row (512 columns of MXFP4, 256 of NVFP4); a row is one CTA of up to
// 1024 threads in the conversion.
bool planes_supported(int fmt, uint32_t H, uint32_t I) {
    const uint32_t unit = fmt == STRATA_MOE_FMT_MXFP4 ? 512u : 256u;
    if (fmt != STRATA_MOE_FMT_MXFP4 && fmt != STRATA_MOE_FMT_NVFP4) return false;
    return H % unit == 0u && I % unit == 0u && H <= kMaxCols && I <= kMaxCols && tensor_map_encoder() != nullptr;
}

// boxes of 16 scale bytes x 128 weight rows
int planes_encode_scale_map(void* out128, int fmt, const void* scales, uint32_t rows, uint32_t K) {
    TensorMapEncodeFn fn = tensor_map_encoder();
    if (!fn) return -1;
    const cuuint64_t row_bytes = fmt == STRATA_MOE_FMT_MXFP4 ? K / 32u : K / 16u;
    const cuuint64_t dims[2] = {row_bytes, rows};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {16u, kMT};
    const cuuint32_t estr[2] = {1, 1};
    return fn(static_cast<CUtensorMap*>(out128), CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(scales), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -1;
}

void launch_rows_to_planes(int fmt, const void* src, bool f32, uint32_t rows, const uint32_t* rows_dev, uint32_t cols,
                           const uint32_t* dest, uint32_t k, const PlaneRows& out, bool settled, cudaStream_t s) {
    if (rows == 0u) return;
    if (fmt == STRATA_MOE_FMT_MXFP4) launch_planes_fmt<STRATA_MOE_FMT_MXFP4>(src, f32, rows, rows_dev, cols, dest, k, out, settled, s);
    else launch_planes_fmt<STRATA_MOE_FMT_NVFP4>(src, f32, rows, rows_dev, cols, dest, k, out, settled, s);
    ++g_kernel_launches;
}

int launch_planes_gate_up(int fmt, const PlaneArgs& a, const void* wmaps, const void* smaps, cudaStream_t s) {
    if (fmt == STRATA_MOE_FMT_MXFP4) return launch_planes_rows<STRATA_MOE_FMT_MXFP4, true>(a, wmaps, smaps, s);
    return launch_planes_rows<STRATA_MOE_FMT_NVFP4, true>(a, wmaps, smaps, s);
}
int launch_planes_down(int fmt, const PlaneArgs& a, const void* wmaps, const void* smaps, cudaStream_t s) {
    if (fmt == STRATA_MOE_FMT_MXFP4) return launch_planes_rows<STRATA_MOE_FMT_MXFP4, false>(a, wmaps, smaps, s);
    return launch_planes_rows<STRATA_MOE_FMT_NVFP4, false>(a, wmaps, smaps, s);
}

}  // namespace smoe
