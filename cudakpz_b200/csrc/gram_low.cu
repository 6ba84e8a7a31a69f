// gram_low.cu -- exact Gram of snapshots whose shifted heights fit one int8 limb (sm_100a).
//
// The snapshots' height ranges are known from when they were added; where every v = h - c lies in
// [-126, 126] (a row's b(y), at most one beyond, then also fits a byte), v is its own int8 operand and
// no tile ever needs the three-limb form of gram_tc.cu.  That removes the need to hand tiles of two kinds to one issuing thread, which is
// what bounded that kernel: at 16384^2 its barrier round trip between eight producers and one
// consumer took 4.5 of its 9.0 ms with nothing built, loaded or multiplied.  Measured on a B200, 64
// snapshots: 16384^2 9.05 -> 3.07 ms, 4096^2 0.76 -> 0.31 ms; what bounds it now is shared memory
// (lookups, row stores and 6 KB of MMA operands per K step: 68 % of its wavefronts at 8192^2) and the
// integer ALU (24 instructions for eight sites of a snapshot, 59 % active).
//
// Here sixteen warps form eight pairs, and a pair does everything for its own contiguous run of
// 128-site tiles (gram_slope.cuh gives the walk): lane l of its two warps walks snapshots l and
// l + 32, writes their 128 values as rows of the K-major SWIZZLE_128B operand into one of
// the pair's two buffers, and after the pair's barrier one thread issues the tile's four MMAs
//   D[0:128, 0:64] += A[0:128] . A[0:64]^T       (kind::i8, signed, M = 128, N = 64, K = 32)
// into the pair's own 64 TMEM columns; their completion frees the buffer.  Pairs share nothing.
// Only 64 of the 128 rows are the tile's: even pairs read it as rows 0-63 (then lanes 0-63 of the
// accumulator are the pair's, which its warps 0 and 1 modulo 4 can load), odd pairs as rows
// 64-127 (lanes 64-127, warps 2 and 3 modulo 4).  The other rows are whatever lies in the
// neighbouring buffer, and their sums are never read.
//
// Four sites per table lookup: the 4-bit pattern of two even and two odd X-slope bits gives the
// four cumulative steps as bytes (biased by 4), added to the broadcast value before them; sixteen
// 4-byte entries lie in sixteen banks, so a warp's lookups never conflict (a 256-entry table of
// eight steps takes about five wavefronts a lookup).
//
// Sums: |v v'| <= r^2 for the largest |v| = r, so an int32 accumulator holds `window` tiles, after
// which (and at the end) the pair's warps add its 64 x 64 block to the int64 result.
#include <algorithm>

#include "gram_mma.cuh"
#include "kpzb_api_internal.h"
#include "kpzb_gram.h"

namespace kpzb {

constexpr int GL_PAIRS = 8;
constexpr int GL_THREADS = GL_PAIRS * 64;
constexpr int GL_BUF = 64 * GS_TILE;  // 8 KB: 64 rows of 128 sites
constexpr int GL_COLS = 64;           // TMEM columns of a pair
constexpr int GL_SMEM = GL_PAIRS * 2 * GL_BUF + 1024;

__device__ __forceinline__ void pair_sync(int pair) { asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory"); }

__global__ void __launch_bounds__(GL_THREADS, 1)
gram_low_kernel(const SlopeSnapGeom g, uint64_t nkt, uint32_t window, unsigned long long* __restrict__ G,
                unsigned int* __restrict__ err)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t empty[GL_PAIRS][2], done[GL_PAIRS];
    __shared__ uint32_t lut[16];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int give_up[GL_PAIRS];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pair = warp >> 1, half = warp & 1;
    const bool lead = half == 0 && lane == 0;

    if (threadIdx.x < GL_PAIRS) {
        mbar_init(&empty[threadIdx.x][0], 1);
        mbar_init(&empty[threadIdx.x][1], 1);
        mbar_init(&done[threadIdx.x], 1);
        give_up[threadIdx.x] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 16) {
        // even-x bits in bits 0-1, odd-x bits in bits 2-3, site order e, o, e, o
        int cum = 4;
        uint32_t w = 0;
        for (int j = 0; j < 4; ++j) {
            cum += 2 * (int)((threadIdx.x >> ((j & 1 ? 2 : 0) + (j >> 1))) & 1u) - 1;
            w |= (uint32_t)cum << (8 * j);
        }
        lut[threadIdx.x] = w;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                     "r"(GL_PAIRS * GL_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t dcol = tmem_base + (uint32_t)(pair * GL_COLS);

    // contiguous tiles [t0, t1) of this pair
    const uint64_t npairs = (uint64_t)gridDim.x * GL_PAIRS, pid = (uint64_t)blockIdx.x * GL_PAIRS + (uint64_t)pair;
    const uint64_t per = nkt / npairs, rem = nkt % npairs;
    const uint64_t t0 = pid * per + (pid < rem ? pid : rem);
    const uint32_t ntiles = (uint32_t)(per + (pid < rem ? 1 : 0));

    const int s = 32 * half + lane;  // this lane's snapshot
    const bool pres = s < g.n;
    const int2* rows = g.rows + (uint64_t)s * g.nrows;
    uint8_t* buf0 = smem + pair * 2 * GL_BUF;
    // MMA operands of the pair's two buffers: B the tile, A the 128 rows that hold it as rows 0-63
    // (even pairs) or 64-127 (odd pairs, whose buffers lie at least two buffers into the array)
    const uint32_t bsm = smem_u32(buf0), asm0 = bsm - (pair & 1 ? GL_BUF : 0);
    const uint32_t idesc = idesc_i8(128, 64);
    const int tpr_lg = g.lx - 7;
    const uint64_t tmask = (1ull << tpr_lg) - 1;

    auto load = [&](uint32_t m) { return pres && m < ntiles ? __ldg(slope_tile(g, s, t0 + m)) : make_uint4(0u, 0u, 0u, 0u); };
    // tiles are fetched two ahead
    uint4 n0 = load(0), n1 = load(1);
    int32_t b = 0, z = 0;            // value before the tile; v(0, y) of its row
    int2 bz_n = make_int2(0, 0);     // {b, z} of the next row
    uint32_t in_window = 0, flushes = 0;
    bool ok = true;

    // add the pair's accumulator to G (all its MMAs issued), both warps; false when a wait expired
    auto flush = [&]() {
        if (lead) {
            umma_commit(&done[pair]);
            if (!mbar_wait_bounded(&done[pair], flushes & 1u)) give_up[pair] = 1;
        }
        ++flushes;
        pair_sync(pair);
        if (give_up[pair]) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c0 = 0; c0 < GL_COLS; c0 += 32) {
            uint32_t v[32];
            const uint32_t taddr = dcol + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)c0;
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                  "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                  "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                : "r"(taddr));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (s <= c0 + j && c0 + j < g.n) atomicAdd(&G[s * 64 + c0 + j], (unsigned long long)(long long)(int32_t)v[j]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        pair_sync(pair);
        return true;
    };

    for (uint32_t m = 0; m < ntiles; ++m) {
        const uint64_t t = t0 + m;
        const uint4 w = n0;
        n0 = n1;
        n1 = load(m + 2);
        const uint64_t y = t >> tpr_lg;
        const uint32_t x0 = (uint32_t)(t & tmask) << 7;
        if ((m == 0 || x0 == 0) && pres) {
            const int2 bz = m == 0 ? __ldg(rows + y) : bz_n;
            if (y + 1 < g.nrows) bz_n = __ldg(rows + y + 1);
            z = bz.y;
            // value before site x0 (plus one at x0 = 0, whose own step is cleared below)
            b = bz.x + 1 + (x0 == 0 ? 0 : 2 * slope_count_before(g, s, y, x0) - (int32_t)x0);
        }
        const int j = (int)(m & 1u);
        if (lead && !mbar_wait_bounded(&empty[pair][j], ((m >> 1) & 1u) ^ 1u)) give_up[pair] = 1;
        pair_sync(pair);
        if (give_up[pair]) {
            ok = false;
            break;
        }
        if (pres) {
            uint8_t* row = buf0 + j * GL_BUF + s * GS_TILE;
            uint32_t base = (uint32_t)(b + 124) * 0x01010101u;  // bytes: value before the four sites, + 124
#pragma unroll
            for (int h = 0; h < 2; ++h) {  // 64 sites: one word of each X quadrant
                uint32_t E = y & 1 ? (h ? w.w : w.z) : (h ? w.y : w.x);
                const uint32_t O = y & 1 ? (h ? w.y : w.x) : (h ? w.w : w.z);
                if (h == 0 && x0 == 0) E &= ~1u;  // x = 0 closes the row in the walk
                // nibble i: pattern of sites 8 i .. 8 i + 3, and of 8 i + 4 .. 8 i + 7
                const uint32_t A = (E & 0x33333333u) | ((O & 0x33333333u) << 2);
                const uint32_t B = ((E >> 2) & 0x33333333u) | (O & 0xCCCCCCCCu);
#pragma unroll
                for (int c = 0; c < 4; ++c) {  // sixteen sites
                    uint32_t out[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint32_t p = i & 1 ? B : A;
                        const int sh = 4 * (2 * c + (i >> 1));
                        const uint32_t off = (sh >= 2 ? p >> (sh - 2) : p << 2) & 0x3Cu;
                        // bytes v + 128: no carry, every v lies in [-128, 127]
                        const uint32_t u = base + *reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(lut) + off);
                        base = __byte_perm(u, 0u, 0x3333) - 0x04040404u;
                        out[i] = u ^ 0x80808080u;
                        b = (int32_t)(u >> 24) - 128;
                    }
                    if (h == 0 && c == 0 && x0 == 0) out[0] = (out[0] & ~0xFFu) | ((uint32_t)z & 0xFFu);
                    *reinterpret_cast<uint4*>(row + (((4 * h + c) ^ (s & 7)) << 4)) = make_uint4(out[0], out[1], out[2], out[3]);
                }
            }
        }
        // the rows are visible to the tensor core before one thread of the pair hands them over
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        pair_sync(pair);
        if (lead) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc0 = in_window ? 1u : 0u;
#pragma unroll
            for (int kk = 0; kk < GS_TILE / 32; ++kk)
                umma_i8(dcol, sdesc_sw128(asm0 + j * GL_BUF + 32 * kk), sdesc_sw128(bsm + j * GL_BUF + 32 * kk), idesc,
                        kk ? 1u : acc0);
            umma_commit(&empty[pair][j]);
        }
        if (++in_window == window && m + 1 < ntiles) {
            ok = flush();
            if (!ok) break;
            in_window = 0;
        }
    }
    if (ok && ntiles > 0) ok = flush();
    if (!ok && lead) {
        atomicExch(err, 1u);
        // bounded: what was issued completes before the accumulator columns are released
        umma_commit(&done[pair]);
        mbar_wait_bounded(&done[pair], flushes & 1u);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(GL_PAIRS * GL_COLS));
}

kpzb_status gram_low_run(const SlopeSnapGeom& g, uint64_t N, int sm_count, int64_t range, unsigned long long* d_g,
                         unsigned int* d_err, int64_t* out, cudaStream_t st)
{
    cudaError_t e = cudaFuncSetAttribute(gram_low_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GL_SMEM);
    if (e != cudaSuccess) return cuda_fail(e, "gram smem attribute");
    if ((e = cudaMemsetAsync(d_g, 0, 64 * 64 * 8, st)) != cudaSuccess) return cuda_fail(e, "memset G");
    if ((e = cudaMemsetAsync(d_err, 0, 4, st)) != cudaSuccess) return cuda_fail(e, "memset flag");
    const int64_t r2 = std::max<int64_t>(1, range * range);
    const uint32_t window = (uint32_t)std::min<int64_t>(0x7FFFFFFF / (r2 * GS_TILE), 1 << 30);
    gram_low_kernel<<<sm_count, GL_THREADS, GL_SMEM, st>>>(g, N / GS_TILE, window, d_g, d_err);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "gram_low_kernel");
    unsigned int flag = 0;
    if ((e = cudaMemcpyAsync(out, d_g, 64 * 64 * 8, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return cuda_fail(e, "G copy");
    if ((e = cudaMemcpyAsync(&flag, d_err, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return cuda_fail(e, "gram flag");
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return cuda_fail(e, "gram sync");
    if (flag) return fail(KPZB_ETIMEOUT, "a bounded device wait in the tensor-core Gram expired");
    return KPZB_OK;
}

}  // namespace kpzb
