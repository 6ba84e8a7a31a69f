// gram_mma.cuh -- what the two tensor-core Gram kernels share (gram_tc.cu, gram_low.cu): bounded
// mbarrier waits, tcgen05 int8 descriptors and issue, and a producer's starting count.
#pragma once
#include <cstdint>

#include "gram_slope.cuh"
#include "scabit_band.cuh"

namespace kpzb {

constexpr uint64_t TC_WAIT_NS = 4000000000ull;    // bound of every mbarrier wait (4 s)

// UMMA instruction descriptor, kind::i8: S32 accumulate (bits 4-5 = 2), signed A and B
// (bits 7-9, 10-12 = 1), both K-major, N>>3 at bit 17, M>>4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_i8(int M, int N)
{
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Shared-memory descriptor of a K-major SWIZZLE_128B operand: rows of 128 bytes, 8-row
// groups 1024 bytes apart (SBO), LBO 16 bytes, descriptor version 1, layout type 2.
__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t saddr)
{
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
           (2ull << 61);
}

__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// waits for the phase with the given parity; false after TC_WAIT_NS of global time
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity)
{
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    for (;;) {
        for (int k = 0; k < 64; ++k)
            if (mbar_try_wait(bar, parity)) return true;
        if (global_ns() - t0 > TC_WAIT_NS) return false;
    }
}

__device__ __forceinline__ void umma_i8(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(dtmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}

__device__ __forceinline__ void umma_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}

// Count of X-slope bits of row y in [1, x0) of one snapshot, by one thread (the running count a
// producer lane starts from when its run of tiles begins inside a row).
__device__ __forceinline__ int32_t slope_count_before(const SlopeSnapGeom& g, int s, uint64_t y, uint32_t x0)
{
    const uint64_t t0 = y << (g.lx - 7);
    int32_t cnt = 0;
    for (uint32_t j = 0; j < (x0 >> 7); ++j) {
        const uint4 v = __ldg(slope_tile(g, s, t0 + j));
        cnt += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
    }
    // site x = 0 (sublattice y & 1, word 0, bit 0) closes the row: not part of the running count
    if (x0 > 0) {
        const uint4 v = __ldg(slope_tile(g, s, t0));
        cnt -= (int32_t)((y & 1 ? v.z : v.x) & 1u);
    }
    return cnt;
}

}  // namespace kpzb
