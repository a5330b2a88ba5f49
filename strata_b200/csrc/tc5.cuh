// Pieces shared by the kernels that run on the 5th-generation tensor cores: barriers with BOUNDED waits, tiled TMA loads,
// shared-memory matrix descriptors, tensor-memory loads and stores, and the position of a ring of stages.
#pragma once
#include <cuda.h>
#include <stdint.h>

namespace smoe {

// The driver's tensor-map encoder, or nullptr (prefill.cu).
typedef CUresult (*TensorMapEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
TensorMapEncodeFn tensor_map_encoder();

constexpr uint32_t kSpinLimit = 1u << 19;   // x up to kWaitHintNs each: about two seconds
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
// Bounded waits: false when the phase did not complete within the limit (about two seconds) or another role raised
// the abort flag.  Each try_wait carries a suspend-time hint: the hardware parks the thread until the phase completes
// or the hint expires.  A polling warp takes issue slots from the decode warps of its scheduler, so tighter polling
// is slower (measured on a 333-token INT4 step: gate/up 1.45 ms as here, 1.69 ms with a four-instruction poll loop).
constexpr uint32_t kWaitHintNs = 4096;
__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(addr), "r"(parity), "r"(kWaitHintNs)
        : "memory");
    return done != 0u;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const volatile uint32_t* abort_flag) {
    const uint32_t addr = smem_u32(bar);
    for (uint32_t spin = 0; spin < kSpinLimit; ++spin) {
        if (mbar_try(addr, parity)) return true;
        if ((spin & 63u) == 63u && *abort_flag) return false;
    }
    return false;
}
// The same for a warp that goes on to warp-wide instructions: lanes may see completion, the time-out or the abort flag at
// different polls, so the loop itself runs on votes and the warp leaves it as one.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, const volatile uint32_t* abort_flag) {
    const uint32_t addr = smem_u32(bar);
    for (uint32_t spin = 0; spin < kSpinLimit; ++spin) {
        if (__all_sync(0xFFFFFFFFu, mbar_try(addr, parity))) return true;
        if ((spin & 63u) == 63u && __any_sync(0xFFFFFFFFu, *abort_flag != 0u)) return false;
    }
    return false;
}
// Barrier 1 over THREADS threads of whole warps; true on every one of them when `failed` is true on any.
template <uint32_t THREADS>
__device__ __forceinline__ bool group_vote(bool failed) {
    uint32_t any;
    __syncwarp();      // the lanes of the polling warp may come out of their wait one by one
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.or.pred q, 1, %2, p;\n selp.u32 %0, 1, 0, q;\n}"
        : "=r"(any)
        : "r"((uint32_t)failed), "n"(THREADS)
        : "memory");
    return any != 0u;
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint32_t x, uint32_t y,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// Contiguous global -> shared copy, addresses and size multiples of 16 bytes.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// Low word of a shared-memory matrix descriptor: start address / 16, leading byte offset unused (1).  K-major operand,
// 128-byte swizzle, 8-row groups 1024 B apart; the high word (kDescHi) holds the stride between the groups / 16, the
// descriptor version of this architecture (bit 46) and the swizzle (2 at bit 61).
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | (1u << 16); }
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);   // see umma_desc_lo
__device__ __forceinline__ bool elect_one() {
    uint32_t e;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xFFFFFFFF;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(e));
    return e != 0u;
}
// This thread's 32 words -> 32 consecutive columns of its tensor-memory lane.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t v[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t v[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// After a wait on copies that an aborting producer issued but nobody may consume: give each a bounded chance to land.
__device__ __forceinline__ void drain_copies(uint64_t* full, uint32_t issued, uint32_t stages) {
    const uint32_t pending = issued < stages ? issued : stages;
    for (uint32_t q = 0; q < pending; ++q) {
        const uint32_t j = issued - 1u - q;
        const uint32_t addr = smem_u32(&full[j % stages]);
        for (uint32_t spin = 0; spin < (1u << 16); ++spin) {
            uint32_t done;
            asm volatile(
                "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                " selp.u32 %0, 1, 0, p;\n}"
                : "=r"(done)
                : "r"(addr), "r"((j / stages) & 1u)
                : "memory");
            if (done) break;
        }
    }
}

// A position in a ring of N stages and the parity its barriers have there.
template <uint32_t N>
struct Ring {
    uint32_t i = 0, ph = 0;
    __device__ __forceinline__ void next(uint32_t step = 1u) {
        i += step;
        if (i >= N) { i -= N; ph ^= 1u; }
    }
};

}  // namespace smoe
