// DSV4-exact numerical mode of the routed expert: the arithmetic of the reference's DeepSeek-V4
// kernels reproduced bit for bit, for hosts that must match a DeepSeek-V4 deployment exactly.
//
//   quantize_activation_e4m3_kernel   kernels/cuda/backend.cu:247-272  (value rule :212-225)
//   deepseek_fp4_gate_up_kernel       kernels/cuda/backend.cu:2308-2376
//   deepseek_fp4_down_kernel          kernels/cuda/backend.cu:2378-2413
//   CPU replay of all three           kernels/cpu/dsv4_fp4_expert.cpp:58-163, 774-884
//   deepseek_fp8_gate_up_kernel / deepseek_fp8_down_kernel (the shared expert: FP8 E4M3 weights, one
//   E8M0 scale per 128 x 128 block)   kernels/cuda/backend.cu:2781-2863
//
// The reference computes one output row with a 256-thread block: thread t accumulates the columns
// t, t + 256, ... in increasing order with sum = fma(x * w, scale, sum), then the block adds the 256
// partial sums in a fixed tree (five shuffle rounds per warp, then the eight warp sums).  The
// result depends on that association, so this kernel keeps it and only changes who computes it:
// ONE warp owns an output row; lane l plays the reference's threads 8l .. 8l+7 (eight
// accumulators per token), which makes every weight load a contiguous 128 bytes per warp; a warp
// works on four weight rows at once (an activation load serves all of them) and two token rows of
// the expert share one pass over the weights.  The reduction tree is evaluated in the same order
// with two shuffle rounds, three in-register rounds and the final three rounds over the eight
// "warp" sums.  Bound by instruction issue and latency (ncu, 4 tokens of 4096 x 2048, 21
// experts with rows: gate/up 156 us, down 83 us, DRAM 15 % busy, issue slots 62 - 64 %, 3.8 warps per
// scheduler, a fifth of their time waiting for loads of token rows and scales): 128 registers leave 16
// warps per SM, each with eight 256-column steps of four rows, 4 KB, on the way.  With 165 registers,
// 12 warps and one step on the way it was 204 us and 107 us, issue slots 42 %.
#include "common.cuh"
#include "libm_exact.cuh"

namespace smoe {

namespace {

__device__ __forceinline__ float bf16_round_dev(float v) {
    uint32_t b = __float_as_uint(v);
    if ((b & 0x7FFFFFFFu) > 0x7F800000u) b = (b | 0x00400000u) & 0xFFFF0000u;
    else b = (b + 0x7FFFu + ((b >> 16) & 1u)) & 0xFFFF0000u;
    return __uint_as_float(b);
}

__device__ __forceinline__ float quantize_e4m3_value_dev(float value) {
    const float magnitude = fminf(fabsf(value), 448.0f);
    float q;
    if (magnitude < 0.015625f) {
        q = __fmul_rn(rintf(__fmul_rn(magnitude, 512.0f)), 0.001953125f);
    } else {
        int e = (int)((__float_as_uint(magnitude) >> 23) & 0xFFu) - 127;   // frexp exponent - 1
        e = max(-6, min(8, e));
        const float step = __uint_as_float((uint32_t)(e - 3 + 127) << 23);
        q = fminf(__fmul_rn(rintf(__fdiv_rn(magnitude, step)), step), 448.0f);
    }
    return copysignf(q, value);
}

// exp2f(ceilf(log2f(maximum / 448))) as the host evaluates it.  log2 is taken in double and rounded
// to float: equal to the host's float log2f except when the true logarithm lies within a quarter
// of a float ulp of a rounding boundary next to an integer.
__device__ __forceinline__ float block_scale_dev(float maximum) {
    if (!(maximum > 0.0f)) return 1.0f;
    const float q = __fdiv_rn(maximum, 448.0f);
    const float l = __double2float_rn(log2((double)q));
    if (!(fabsf(l) <= 3.0e38f)) return l > 0.0f ? l : 0.0f;
    return ldexpf(1.0f, (int)ceilf(l));
}

__device__ __forceinline__ float e8m0_dsv4(uint32_t bits) {
    return __uint_as_float(bits == 0xFFu ? 0x7FC00000u : (bits == 0u ? 0x00400000u : bits << 23));
}

// 8 E2M1 nibbles (low nibble = even column) -> 8 floats, 0x8 -> -0.0 like the host table.
__device__ __forceinline__ void e2m1x8_f32(uint32_t w, float v[8]) {
    uint32_t h[4];
    asm("{\n .reg .b8 b0, b1, b2, b3;\n mov.b32 {b0, b1, b2, b3}, %4;\n"
        " cvt.rn.f16x2.e2m1x2 %0, b0;\n cvt.rn.f16x2.e2m1x2 %1, b1;\n"
        " cvt.rn.f16x2.e2m1x2 %2, b2;\n cvt.rn.f16x2.e2m1x2 %3, b3;\n}"
        : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
        : "r"(w));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __half2 p = *reinterpret_cast<const __half2*>(&h[i]);
        v[2 * i] = __low2float(p);
        v[2 * i + 1] = __high2float(p);
    }
}

// 8 E4M3 bytes (two 32-bit words, byte q = column q) -> 8 floats, exact; 0x7F / 0xFF -> NaN.
__device__ __forceinline__ void e4m3x8_f32(uint2 w, float v[8]) {
    const uint32_t words[2] = {w.x, w.y};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        uint32_t lo, hi;
        asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(lo) : "h"((unsigned short)(words[i] & 0xFFFFu)));
        asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(hi) : "h"((unsigned short)(words[i] >> 16)));
        const __half2 a = *reinterpret_cast<const __half2*>(&lo), b = *reinterpret_cast<const __half2*>(&hi);
        v[4 * i] = __low2float(a);
        v[4 * i + 1] = __high2float(a);
        v[4 * i + 2] = __low2float(b);
        v[4 * i + 3] = __high2float(b);
    }
}

// The reference's block tree over the 256 partial sums, held as v[s] on lane l = thread 8l + s.
// Returns the block sum on lane 0.
__device__ __forceinline__ float block_tree(float v[8], uint32_t lane) {
    (void)lane;
#pragma unroll
    for (int s = 0; s < 8; ++s) v[s] = __fadd_rn(v[s], __shfl_down_sync(0xFFFFFFFFu, v[s], 2));  // thread + 16
#pragma unroll
    for (int s = 0; s < 8; ++s) v[s] = __fadd_rn(v[s], __shfl_down_sync(0xFFFFFFFFu, v[s], 1));  // thread + 8
#pragma unroll
    for (int s = 0; s < 4; ++s) v[s] = __fadd_rn(v[s], v[s + 4]);                               // thread + 4
    v[0] = __fadd_rn(v[0], v[2]);
    v[1] = __fadd_rn(v[1], v[3]);
    float w = __fadd_rn(v[0], v[1]);            // warp sum of reference warp l / 4, valid on lanes 0, 4, .., 28
    w = __fadd_rn(w, 0.0f);                     // the rounds that add the zeroed lanes 8..31
    w = __fadd_rn(w, __shfl_down_sync(0xFFFFFFFFu, w, 16));   // warp + 4
    w = __fadd_rn(w, __shfl_down_sync(0xFFFFFFFFu, w, 8));    // warp + 2
    w = __fadd_rn(w, __shfl_down_sync(0xFFFFFFFFu, w, 4));    // warp + 1
    return w;
}

}  // namespace

// ------------------------------------------------------------------------------ quantise
// One warp per (row, 128-column block).  dst row pos <- src row (perm ? perm[pos] / k_div : pos).
__global__ void __launch_bounds__(256) dsv4_quantize_kernel(const float* __restrict__ src,
                                                            const uint32_t* __restrict__ perm, uint32_t k_div,
                                                            uint32_t rows, uint32_t cols, float* __restrict__ dst,
                                                            uint32_t* tiny) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t blocks = (cols + 127u) / 128u;
    const size_t task = (size_t)blockIdx.x * 8u + (threadIdx.x >> 5);
    if (task >= (size_t)rows * blocks) return;
    const uint32_t pos = (uint32_t)(task / blocks), begin = (uint32_t)(task % blocks) * 128u;
    const uint32_t srow = perm ? perm[pos] / k_div : pos;
    const float* s = src + (size_t)srow * cols + begin;
    float* d = dst + (size_t)pos * cols + begin;
    float x[4];
    float mx = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t c = lane + 32u * i;
        x[i] = begin + c < cols ? s[c] : 0.0f;
        mx = fmaxf(mx, fabsf(x[i]));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, off));
    const float scale = block_scale_dev(mx);
    // below 2^-120 or above 2^109: see dsv4_rows
    if (tiny != nullptr && lane == 0 && mx > 0.0f && !(scale >= 7.5e-37f && scale <= 6.4e32f)) *tiny = 1u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t c = lane + 32u * i;
        if (begin + c < cols) d[c] = __fmul_rn(quantize_e4m3_value_dev(__fdiv_rn(x[i], scale)), scale);
    }
}

// ------------------------------------------------------------------------------ matvec rows
struct Dsv4Args {
    uint32_t n_groups, K, R;
    const uint32_t* offsets;
    WeightTable w0, w1;        // gate, up  (DUAL)  or  down, unused
    const float* x;            // [pairs, K] fp32, already E4M3-quantised
    const float* coef;         // [pairs] or nullptr (= 1)
    float limit;
    float* out;                // [pairs, R]
    uint32_t* status;
    const uint32_t* tiny;      // nonzero: activations so small or large were seen that x * w may round or overflow (or nullptr: assume so)
};

constexpr uint32_t kDsv4Warps = 4, kDsv4Ctas = 4;   // warps per CTA, CTAs per SM (128 registers a thread: a few spills with two token rows, made up for by a third more warps)
constexpr uint32_t kDsv4MaxGroups = 1024;
constexpr uint32_t kDsv4Ahead = 8;      // steps of 256 columns that the weight copies run ahead

// One warp, RW weight rows (DUAL: RW / 2 gate rows and the same up rows), NTOK token rows at `pos0` (only `cnt` of them
// exist; the others repeat the last one and are dropped).
//
// The reference's step is sum = fma(x * w, scale, sum).  x has four significant bits, w two (FP4) or four (FP8) and
// scale is a power of two, so x * w and w * scale are both exact and fma(x, w * scale, sum) rounds the same exact
// number: one multiply per weight instead of one per weight and token.  That needs w * scale finite (6 * 2^(byte - 127)
// for FP4, 448 * 2^(byte - 127) for FP8: bytes below 250 / 247) and x * w neither below the subnormal grid nor beyond the
// largest float (x is at most 448 block scales and w at most 448: scales up to 2^109); all are checked and the chunk
// takes the reference's two steps otherwise.
template <bool DUAL, bool FP8, int RW, int NTOK>
__device__ __forceinline__ void dsv4_rows(const Dsv4Args& a, uint32_t g, uint32_t row, size_t pos0, uint32_t cnt,
                                          bool two_step, uint32_t lane, uint32_t* ring, bool& bad) {
    const uint32_t K = a.K;
    constexpr int HALF = DUAL ? RW / 2 : RW;
    const uint8_t *p[RW], *s[RW];
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        const uint32_t rr = row + (uint32_t)(r % HALF);
        const WeightTable& w = DUAL && r >= HALF ? a.w1 : a.w0;
        p[r] = w.packed[g] + (FP8 ? (size_t)rr * K : (size_t)rr * (K / 2u)) + lane * (FP8 ? 8u : 4u);
        s[r] = w.scales[g] + (FP8 ? (size_t)(rr / 128u) * ((K + 127u) / 128u) : (size_t)rr * (K / 32u));
    }
    const float* xr[NTOK];
#pragma unroll
    for (int k = 0; k < NTOK; ++k) xr[k] = a.x + (pos0 + min((uint32_t)k, cnt - 1u)) * K + lane * 8u;
    float acc[RW][NTOK][8];
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
        for (int k = 0; k < NTOK; ++k)
#pragma unroll
            for (int q = 0; q < 8; ++q) acc[r][k][q] = 0.0f;
    // Weights come through a ring in shared memory, kDsv4Ahead steps of 256 columns ahead, by asynchronous copies: every lane
    // fetches and reads its own words, so a wait for its copies is all the synchronisation.  A warp's four rows are 512 bytes a
    // step; with one step ahead, in registers, an SM had 6 KB in flight and streamed 1.5 TB/s over the GPU (three steps more
    // in registers spilled and were slower).  A row's scales share one cache line: one step ahead in registers.
    constexpr uint32_t kWords = FP8 ? 2u : 1u;
    uint32_t sq[RW];
    auto fetch = [&](uint32_t slot, uint32_t c) {
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(ring + ((slot * RW + r) * 32u + lane) * kWords);
            if (FP8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(p[r] + c) : "memory");
            else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(p[r] + c / 2u) : "memory");
        }
    };
    auto scales = [&](uint32_t c) {
#pragma unroll
        for (int r = 0; r < RW; ++r) sq[r] = __ldg(s[r] + (c + lane * 8u) / (FP8 ? 128u : 32u));
    };
    const uint32_t end = K > lane * 8u ? K - lane * 8u : 0u;   // this lane's columns start below K
#pragma unroll
    for (uint32_t i = 0; i < kDsv4Ahead; ++i) {
        if (256u * i < end) fetch(i, 256u * i);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // the token rows (from L1 and L2) are requested a step ahead as well where registers allow it: one row
    constexpr bool kNext = NTOK == 1;
    float4 xa[NTOK], xb[NTOK];
    auto tokens = [&](uint32_t c) {
#pragma unroll
        for (int k = 0; k < NTOK; ++k) {
            xa[k] = __ldg(reinterpret_cast<const float4*>(xr[k] + c));
            xb[k] = __ldg(reinterpret_cast<const float4*>(xr[k] + c) + 1);
        }
    };
    if (end) scales(0);
    if (kNext && end) tokens(0);
    uint32_t slot = 0;
    for (uint32_t c = 0; c < end; c += 256u) {
        float xv[NTOK][8];
        if (!kNext) tokens(c);
#pragma unroll
        for (int k = 0; k < NTOK; ++k) {
            xv[k][0] = xa[k].x; xv[k][1] = xa[k].y; xv[k][2] = xa[k].z; xv[k][3] = xa[k].w;
            xv[k][4] = xb[k].x; xv[k][5] = xb[k].y; xv[k][6] = xb[k].z; xv[k][7] = xb[k].w;
        }
        if (kNext && c + 256u < end) tokens(c + 256u);
        asm volatile("cp.async.wait_group %0;" ::"n"(kDsv4Ahead - 1u) : "memory");
        uint2 w[RW];
        uint32_t sb[RW];
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            const volatile uint32_t* at = ring + ((slot * RW + r) * 32u + lane) * kWords;
            w[r].x = at[0];
            if (FP8) w[r].y = at[1];
            sb[r] = sq[r];
        }
        if (c + 256u * kDsv4Ahead < end) fetch(slot, c + 256u * kDsv4Ahead);
        asm volatile("cp.async.commit_group;" ::: "memory");
        slot = slot + 1u == kDsv4Ahead ? 0u : slot + 1u;
        if (c + 256u < end) scales(c + 256u);
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            float wv[8];
            if (FP8) e4m3x8_f32(w[r], wv);
            else e2m1x8_f32(w[r].x, wv);
            const float sc = e8m0_dsv4(sb[r]);
            if (two_step || sb[r] >= (FP8 ? 247u : 250u)) {
#pragma unroll
                for (int k = 0; k < NTOK; ++k)
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        acc[r][k][q] = __fmaf_rn(__fmul_rn(xv[k][q], wv[q]), sc, acc[r][k][q]);
            } else {
#pragma unroll
                for (int q = 0; q < 8; ++q) wv[q] = __fmul_rn(wv[q], sc);
#pragma unroll
                for (int k = 0; k < NTOK; ++k)
#pragma unroll
                    for (int q = 0; q < 8; ++q) acc[r][k][q] = __fmaf_rn(xv[k][q], wv[q], acc[r][k][q]);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < NTOK; ++k) {
        if ((uint32_t)k >= cnt) break;      // uniform across the warp
        const size_t pos = pos0 + k;
#pragma unroll
        for (int r = 0; r < HALF; ++r) {
            const float t0 = block_tree(acc[r][k], lane);
            if (DUAL) {
                const float t1 = block_tree(acc[r + (DUAL ? HALF : 0)][k], lane);
                if (lane == 0) {
                    const float g_r = bf16_round_dev(t0), u_r = bf16_round_dev(t1);
                    if (!(fabsf(g_r) <= 3.0e38f) || !(fabsf(u_r) <= 3.0e38f)) bad = true;
                    const float lg = fminf(g_r, a.limit);
                    const float lu = fmaxf(-a.limit, fminf(u_r, a.limit));
                    const float gt = __uint_as_float(__float_as_uint(lg) & 0xFFFF0000u);  // table index = top 16 bits
                    const float silu = (fabsf(gt) <= 3.0e38f) ? __fmul_rn(gt, sigmoid_two_branch(gt)) : gt;
                    float act = __fmul_rn(silu, lu);
                    act = __fmul_rn(act, a.coef ? a.coef[pos] : 1.0f);
                    a.out[pos * a.R + row + r] = bf16_round_dev(act);
                }
            } else if (lane == 0) {
                a.out[pos * a.R + row + r] = bf16_round_dev(t0);
            }
        }
    }
}

// FP8 = false: E2M1 nibbles + one E8M0 scale per 32 columns of a row.
// FP8 = true : E4M3 bytes + one E8M0 scale per 128 x 128 block (scales [ceil(R / 128), ceil(K / 128)]).
//
// A warp takes four output rows of one expert with rows (gate/up: two of each).  Every CTA first compacts the list of
// experts that have rows: walking all of them cost a chain of offset loads per empty expert and left most warps of a
// small step with nothing else (4 tokens of 4096 x 2048 x 256 experts, 22 with rows: 0.86 ms per step before).
template <bool DUAL, bool FP8>
__global__ void __launch_bounds__(kDsv4Warps * 32, kDsv4Ctas) dsv4_rows_kernel(Dsv4Args a) {
    __shared__ __align__(16) uint32_t rings[kDsv4Warps][kDsv4Ahead * 4u * 32u * (FP8 ? 2u : 1u)];   // one per warp
    __shared__ uint16_t list[kDsv4MaxGroups];
    __shared__ uint32_t warp_base[kDsv4Warps + 1];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const bool two_step = a.tiny == nullptr || *a.tiny != 0u;
    bool bad = false;
    for (uint32_t g0 = 0; g0 < a.n_groups; g0 += kDsv4MaxGroups) {
        const uint32_t ng = min(kDsv4MaxGroups, a.n_groups - g0);
        // ordered compaction: warp w scans groups [w * span, (w + 1) * span)
        const uint32_t span = (ng + kDsv4Warps - 1u) / kDsv4Warps;
        uint32_t mine = 0;
        for (uint32_t q = 0; q < span; q += 32u) {
            const uint32_t g = warp * span + q + lane;
            const bool has = q + lane < span && g < ng && a.offsets[g0 + g + 1] != a.offsets[g0 + g];
            mine += __popc(__ballot_sync(0xFFFFFFFFu, has));
        }
        if (lane == 0) warp_base[warp + 1u] = mine;
        __syncthreads();
        if (threadIdx.x == 0) {
            warp_base[0] = 0;
            for (uint32_t w = 0; w < kDsv4Warps; ++w) warp_base[w + 1u] += warp_base[w];
        }
        __syncthreads();
        uint32_t at = warp_base[warp];
        for (uint32_t q = 0; q < span; q += 32u) {
            const uint32_t g = warp * span + q + lane;
            const bool has = q + lane < span && g < ng && a.offsets[g0 + g + 1] != a.offsets[g0 + g];
            const uint32_t b = __ballot_sync(0xFFFFFFFFu, has);
            if (has) list[at + __popc(b & ((1u << lane) - 1u))] = (uint16_t)g;
            at += __popc(b);
        }
        __syncthreads();
        constexpr uint32_t RB = DUAL ? 2u : 4u;      // output rows per task (R is a multiple of 128)
        const uint32_t per = a.R / RB, total = warp_base[kDsv4Warps] * per;
        for (uint32_t task = blockIdx.x * kDsv4Warps + warp; task < total; task += gridDim.x * kDsv4Warps) {
            const uint32_t slot = task / per, row = (task - slot * per) * RB;
            const uint32_t g = g0 + list[slot];
            const uint32_t row0 = a.offsets[g], cnt = a.offsets[g + 1] - row0;
            for (uint32_t tb = 0; tb < cnt;) {
                const uint32_t left = cnt - tb;
                if (left == 1u) {
                    dsv4_rows<DUAL, FP8, 4, 1>(a, g, row, (size_t)row0 + tb, 1u, two_step, lane, rings[warp], bad);
                    tb += 1u;
                } else {
                    dsv4_rows<DUAL, FP8, 4, 2>(a, g, row, (size_t)row0 + tb, min(2u, left), two_step, lane, rings[warp], bad);
                    tb += 2u;
                }
            }
        }
        __syncthreads();     // the list is rebuilt for the next block of groups
    }
    if (bad) atomicOr(a.status, kStatusNonFiniteOutput);
}

// ------------------------------------------------------------------------------ join
// out[t] = bf16(sum_r y[inv[t * k + r]] + bf16(shared[t])): the routed rows (already BF16-rounded, route
// weight already applied) are added in selection-rank order starting from +0, the shared row is
// rounded on its own, then the total is rounded (src/models/dsv4/deepseek_runtime.cpp:5897-5914;
// device form kernels/cuda/backend.cu:2868-2880).
__global__ void __launch_bounds__(256) dsv4_join_kernel(const float* __restrict__ y, const uint32_t* __restrict__ inv,
                                                        const float* __restrict__ shared, uint32_t T, uint32_t k,
                                                        uint32_t H, float* __restrict__ out, uint32_t* status) {
    bool bad = false;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < (size_t)T * H;
         i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t t = (uint32_t)(i / H), c = (uint32_t)(i % H);
        float o = 0.0f;
        for (uint32_t r = 0; r < k; ++r) {
            const uint32_t pos = inv[(size_t)t * k + r];
            if (pos == 0xFFFFFFFFu) continue;
            o = __fadd_rn(o, bf16_round_dev(y[(size_t)pos * H + c]));
        }
        const float sh = shared ? bf16_round_dev(shared[i]) : 0.0f;
        o = bf16_round_dev(__fadd_rn(o, sh));
        bad |= !(fabsf(o) <= 3.0e38f);
        out[i] = o;
    }
    if (bad) atomicOr(status, kStatusNonFiniteOutput);
}

void launch_dsv4_join(const float* y, const uint32_t* inv, const float* shared, uint32_t T, uint32_t k, uint32_t H,
                      float* out, uint32_t* status, cudaStream_t s) {
    if (T == 0) return;
    const size_t n = (size_t)T * H;
    const unsigned grid = (unsigned)((n + 255) / 256 < (size_t)kNumSMs * 8u ? (n + 255) / 256 : (size_t)kNumSMs * 8u);
    dsv4_join_kernel<<<grid, 256, 0, s>>>(y, inv, shared, T, k, H, out, status);
    ++g_kernel_launches;
}

// ------------------------------------------------------------------------------ launchers
void launch_dsv4_quantize(const float* src, const uint32_t* perm, uint32_t k_div, uint32_t rows, uint32_t cols,
                          float* dst, cudaStream_t s, uint32_t* tiny) {
    if (rows == 0 || cols == 0) return;
    const size_t tasks = (size_t)rows * ((cols + 127u) / 128u);
    dsv4_quantize_kernel<<<(unsigned)((tasks + 7) / 8), 256, 0, s>>>(src, perm, k_div, rows, cols, dst, tiny);
    ++g_kernel_launches;
}

// a full house of resident CTAs walks the tasks; fewer CTAs when even a full house of groups has fewer tasks
static unsigned dsv4_grid(size_t tasks) {
    const size_t ctas = (tasks + kDsv4Warps - 1) / kDsv4Warps;
    return (unsigned)(ctas < (size_t)kNumSMs * kDsv4Ctas ? ctas : (size_t)kNumSMs * kDsv4Ctas);
}

void launch_dsv4_gate_up(uint32_t n_groups, const uint32_t* offsets, uint32_t H, uint32_t I, const WeightTable& gate,
                         const WeightTable& up, const float* xq, const float* coef, float limit, float* act,
                         uint32_t* status, cudaStream_t s, const uint32_t* tiny, bool fp8) {
    Dsv4Args a{n_groups, H, I, offsets, gate, up, xq, coef, limit, act, status, tiny};
    const unsigned grid = dsv4_grid((size_t)n_groups * (I / 2u));
    if (fp8) dsv4_rows_kernel<true, true><<<grid, kDsv4Warps * 32, 0, s>>>(a);
    else dsv4_rows_kernel<true, false><<<grid, kDsv4Warps * 32, 0, s>>>(a);
    ++g_kernel_launches;
}

void launch_dsv4_down(uint32_t n_groups, const uint32_t* offsets, uint32_t H, uint32_t I, const WeightTable& down,
                      const float* actq, float* y, uint32_t* status, cudaStream_t s, const uint32_t* tiny, bool fp8) {
    Dsv4Args a{n_groups, I, H, offsets, down, down, actq, nullptr, 0.0f, y, status, tiny};
    const unsigned grid = dsv4_grid((size_t)n_groups * (H / 4u));
    if (fp8) dsv4_rows_kernel<false, true><<<grid, kDsv4Warps * 32, 0, s>>>(a);
    else dsv4_rows_kernel<false, false><<<grid, kDsv4Warps * 32, 0, s>>>(a);
    ++g_kernel_launches;
}

}  // namespace smoe
