// dt.cu -- double-tiling (DT) random-sequential dynamics on ENC_LOCAL lattices (sm_100a).
//
// Reference behaviour: SchedulerDT::doMcs (kpz/schedulerDT.cu:38-78) -- per MCS a random
// origin in [0, 2*block) and a shuffled order of the four domain sets, one launch per set;
// kpzKernelTemplateDT + copyInDT/copyOutDT (kpz/kpz.cu:126-155, kpz/kpzCopy.cu:144-187) --
// each block is copied with a one-word halo into shared memory, updated, copied back; the
// inner single-hit double tiling of KpzCores::BaseDT
// (kpz/kpzSimulationPrimitivesTemplates.cu:110-141) -- per attempt round the whole block
// uses one random quadrant (sub-cell) of every thread cell, so the sites updated in a round
// never share a word and need no atomics; the per-site rule of PQSyncRng
// (kpz/kpzSimulationPrimitivesTemplates.cu:229-268).
//
// Geometry: blocks of 256x128 sites (64x32 words) in 32x16 cells of 8x8 sites, 64 rounds per
// launch with one attempt per cell and round (one attempt per site per MCS).  All random
// numbers come from the counter stream (see oracle/kpz_oracle.h), so the CPU emulations
// ko_dt_mcs* reproduce every lattice bit for bit.
//
// The reference's other block-level decompositions (KPZ_INNER_DD, kpz/kpzConst.h:26-35) are
// template parameters: DTDBSH, DB, DBSH (the reference's default) and DBSHRep; and the
// reference's DB4 scheduler (Kpz::Scheduler<Rng, LocalLayoutDB4>,
// kpz/scheduler.cu:37-52, kpz/kpz.cu:95-117): per MCS two launches over every block from a
// random origin in [0, block), no halo, sites within 5 of the block's far edges dead, 32
// BaseDT rounds per launch (kpz/kpzSimulationPrimitivesTemplates.cu:74-103).
#include <cmath>
#include <type_traits>
#include <cstring>

#include "kpzb_api_internal.h"
#include "kpzb_common.cuh"
#include "kpzb_internal.h"

namespace kpzb {

constexpr uint32_t TAG_DT_SUB = 4u;
constexpr uint32_t TAG_DT_POS = 5u;
constexpr uint32_t TAG_DBSH_ORIGIN = 7u;
constexpr uint32_t TAG_DBSH_POS = 8u;
constexpr uint32_t TAG_REP_ORIGIN = 9u;
constexpr uint32_t TAG_REP_POS = 10u;
constexpr uint32_t TAG_REP_U = 11u;
constexpr uint32_t TAG_DB4_ORIGIN = 12u;
constexpr uint32_t TAG_DB4_SUB = 13u;
constexpr uint32_t TAG_DB4_POS = 14u;
constexpr uint32_t TAG_DB4_U = 15u;
constexpr int DT_BXW = 64, DT_BYW = 32;                // block in words
constexpr int DT_BX = 4 * DT_BXW, DT_BY = 4 * DT_BYW;  // block in sites
constexpr int DT_CX = DT_BX / 8, DT_CY = DT_BY / 8;    // block in cells
constexpr int DT_CELLS = DT_CX * DT_CY;
constexpr int DT_ROUNDS = 64;

// Philox key schedule by value: every round key is then a constant-bank operand of the round's
// three-input XOR (3 % to 6 % of these kernels' time where an attempt draws its acceptance; no
// difference to the SCABit kernels).
struct DtKey {
    uint32_t k0[10], k1[10];
};
inline DtKey make_dt_key(Key key)
{
    DtKey k;
    for (uint32_t r = 0; r < 10; ++r) {
        k.k0[r] = key.k0 + r * 0x9E3779B9u;
        k.k1[r] = key.k1 + r * 0xBB67AE85u;
    }
    return k;
}
__device__ __forceinline__ uint4 philox_dt(uint4 c, const DtKey& k)
{
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint64_t p0 = (uint64_t)0xD2511F53u * c.x, p1 = (uint64_t)0xCD9E8D57u * c.z;
        c = make_uint4((uint32_t)(p1 >> 32) ^ c.y ^ k.k0[r], (uint32_t)p1, (uint32_t)(p0 >> 32) ^ c.w ^ k.k1[r], (uint32_t)p0);
    }
    return c;
}

__device__ __forceinline__ uint32_t pick4(const uint4& v, int i)
{
    return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
}

// The rule's acceptance limits for the plain rates: a deposition candidate flips when
// ok_p and its acceptance word u <= lim_p = T_p - 1, likewise q.
struct DtRule {
    bool ok_p, ok_q;
    uint32_t lim_p, lim_q;
};
__device__ __forceinline__ DtRule make_rule(Thresh tp, Thresh tq)
{
    return DtRule{tp.always || tp.planes, tq.always || tq.planes, tp.always ? 0xFFFFFFFFu : tp.t - 1u,
                  tq.always ? 0xFFFFFFFFu : tq.t - 1u};
}

// bytes each holding v, and the sum of two words' bytes modulo 256
__device__ __forceinline__ uint32_t bytes4(uint32_t v) { return 0x01010101u * v; }
__device__ __forceinline__ uint32_t add_bytes(uint32_t a, uint32_t b)
{
    return ((a & 0x7F7F7F7Fu) + (b & 0x7F7F7F7Fu)) ^ ((a ^ b) & 0x80808080u);
}

// Even bits of each byte of v as the byte's low nibble, and back.
__device__ __forceinline__ uint32_t even_nibbles(uint32_t v)
{
    v &= 0x55555555u;
    v = (v | (v >> 1)) & 0x33333333u;
    return (v | (v >> 2)) & 0x0F0F0F0Fu;
}
__device__ __forceinline__ uint32_t spread_nibbles(uint32_t v)
{
    v = (v | (v << 2)) & 0x33333333u;
    return (v | (v << 1)) & 0x55555555u;
}

// The scattered-site kernel keeps a block and its halo (65 x 33 words, 260 x 132 sites) as two bit
// planes in shared memory, the x-slopes and the y-slopes, row by row: 32 sites a word.  One
// address then serves an attempt: x-slopes of the site and its right neighbour from a funnel
// shift of two adjacent words, y-slopes of the site and its lower neighbour one row apart.  Rows
// are 9 words (257 sites and the rest of the halo words), so that the eight rows and eight words a
// warp's cells reach lie at most two to a bank.
constexpr int PL_W = 9, PL_H = 4 * (DT_BYW + 1);
constexpr int PL_WORDS = PL_W * PL_H;

// 4 x 4 byte transpose.
__device__ __forceinline__ void transpose_bytes(const uint32_t a[4], uint32_t o[4])
{
    const uint32_t l0 = __byte_perm(a[0], a[1], 0x5140), l1 = __byte_perm(a[2], a[3], 0x5140);
    const uint32_t h0 = __byte_perm(a[0], a[1], 0x7362), h1 = __byte_perm(a[2], a[3], 0x7362);
    o[0] = __byte_perm(l0, l1, 0x5410);
    o[1] = __byte_perm(l0, l1, 0x7632);
    o[2] = __byte_perm(h0, h1, 0x5410);
    o[3] = __byte_perm(h0, h1, 0x7632);
}

// Block words from (wx0, wy0) on, halo included, to / from two bit planes; `plane` holds the planes
// of the words' even bits and, PL_WORDS on, of their odd bits.  Item i: eight words of one word
// row (or the halo word at its end), i.e. one plane word of four rows.
__device__ __forceinline__ void planes_load(const uint32_t* __restrict__ sys, uint32_t* plane, int tid, int nthreads,
                                            uint32_t wx0, uint32_t wy0, uint32_t Wx, uint32_t Wy)
{
    for (int i = tid; i < (DT_BYW + 1) * PL_W; i += nthreads) {
        const uint32_t r = i / PL_W, g = i - r * PL_W;
        const uint32_t* row = sys + (size_t)((wy0 + r) & (Wy - 1)) * Wx;
        uint32_t w[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) w[k] = (k == 0 || g < 8) ? row[(wx0 + 8 * g + k) & (Wx - 1)] : 0u;
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            uint32_t a[4], o[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) a[k] = even_nibbles(w[2 * k] >> b) | (even_nibbles(w[2 * k + 1] >> b) << 4);
            transpose_bytes(a, o);
#pragma unroll
            for (int k = 0; k < 4; ++k) plane[b * PL_WORDS + (4 * r + k) * PL_W + g] = o[k];
        }
    }
}

__device__ __forceinline__ void planes_store(uint32_t* __restrict__ sys, const uint32_t* plane, int tid, int nthreads,
                                             uint32_t wx0, uint32_t wy0, uint32_t Wx, uint32_t Wy)
{
    for (int i = tid; i < (DT_BYW + 1) * PL_W; i += nthreads) {
        const uint32_t r = i / PL_W, g = i - r * PL_W;
        uint32_t* row = sys + (size_t)((wy0 + r) & (Wy - 1)) * Wx;
        uint32_t w[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            uint32_t a[4], o[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) o[k] = plane[b * PL_WORDS + (4 * r + k) * PL_W + g];
            transpose_bytes(o, a);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                w[2 * k] |= spread_nibbles(a[k] & 0x0F0F0F0Fu) << b;
                w[2 * k + 1] |= spread_nibbles((a[k] >> 4) & 0x0F0F0F0Fu) << b;
            }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (k == 0 || g < 8) row[(wx0 + 8 * g + k) & (Wx - 1)] = w[k];
    }
}

// One attempt of the random-sequential rule (PQSyncRng::update,
// kpz/kpzSimulationPrimitivesTemplates.cu:229-281) at site (x, y) of the planes, in two halves so
// that a thread's attempts of one pass load together: their sites are never neighbours, so
// none of them reads a bit another one flips.
template <bool DIS>
struct DtSite {
    uint32_t* a;
    uint32_t x, x0, x1, y0, y1, d0, d1;
    // x: the site's column (modulo 32), off: the byte offset of its word in a plane
    __device__ __forceinline__ void load(uint32_t* plane, uint32_t x_, uint32_t off)
    {
        x = x_;
        a = reinterpret_cast<uint32_t*>(reinterpret_cast<char*>(plane) + off);
        x0 = a[0];
        x1 = a[1];
        y0 = a[PL_WORDS];
        y1 = a[PL_WORDS + PL_W];
        if (DIS) {
            d0 = a[2 * PL_WORDS];
            d1 = a[3 * PL_WORDS];
        }
    }
    template <bool COUNT>
    __device__ __forceinline__ void flip(uint32_t u, const DtRule& rule, const uint2* rates,
                                         unsigned long long& ndep, unsigned long long& ndes) const
    {
        // bit 0 (bit 1): x-slope of the site (of its right neighbour); bit 0 of ys, yd: y-slope of the
        // site and of its lower neighbour.  A deposition candidate has 0, 1 | 0, 1, a
        // desorption candidate 1, 0 | 1, 0.
        const uint32_t xs = __funnelshift_r(x0, x1, x), ys = __funnelshift_r(y0, y0, x), yd = __funnelshift_r(y1, y1, x);
        const uint32_t cand = (xs ^ (xs >> 1)) & ~(xs ^ ys) & (ys ^ yd) & 1u;
        const bool is_q = (xs & 1u) != 0u;
        bool ok;
        if (DIS) {
            const uint32_t cls = (__funnelshift_r(d0, d0, x) & 1u) | ((__funnelshift_r(d1, d1, x) & 1u) << 1);
            const uint2 r = rates[2u * cls + (is_q ? 1u : 0u)];
            ok = r.x && u <= r.y;
        } else {
            ok = (is_q ? rule.ok_q : rule.ok_p) && u <= (is_q ? rule.lim_q : rule.lim_p);
        }
        if (cand && ok) {
            // other attempts of the pass may flip other bits of these words
            const uint32_t m = __funnelshift_l(1u, 1u, x);
            atomicXor(a, m * 3u);
            if (m >> 31) atomicXor(a + 1, 1u);
            atomicXor(a + PL_WORDS, m);
            atomicXor(a + PL_WORDS + PL_W, m);
            if (COUNT) {
                if (is_q) ++ndes;
                else ++ndep;
            }
        }
    }
};

// Positions of four rounds, a byte each: cell offset px in bits 0-2, py in bits 3-5.  Bit 7 of each
// byte of the result is CLEAR where the attempt's right neighbour site is the one attempted by
// the cell to the right (position `right`) or its lower neighbour site the one attempted by the
// cell below (position `below`).
__device__ __forceinline__ uint32_t not_adjacent(uint32_t pos, uint32_t right, uint32_t below)
{
    // right: px = 7 against 0 and the same py; below: py = 7 against 0 and the same px
    const uint32_t r = (((pos ^ right) & 0x3F3F3F3Fu) ^ 0x07070707u) | (~pos & 0x07070707u);
    const uint32_t d = (((pos ^ below) & 0x3F3F3F3Fu) ^ 0x38383838u) | (~pos & 0x38383838u);
    return (r + 0x7F7F7F7Fu) & (d + 0x7F7F7F7Fu);
}

// DIS: quenched disorder (Disorder2SyncRng_shared, kpz/kpzSimulationPrimitivesTemplates.cu:
// 295-382): dis holds every site's 2-bit rate class in ENC_LOCAL words, copied into a second
// pair of planes; the class picks dr.tp[c] / dr.tq[c].
// SCHEME (the reference's KPZ_INNER_DD, kpz/kpzConst.h:26-35):
//   DT_SCHEME_DTDBSH  single-hit double tiling with a block-wide random offset of the cells per round
//   DT_SCHEME_DBSH    single-hit dead border, borders delayed to later phases of the round
//   DT_SCHEME_DB      the dead-border phases without the per-round cell offset
//   DT_SCHEME_DBSHREP DBSH with the border hits replaced by fresh attempts after the rounds
//
// The dead-border schemes order a round's attempts in three phases: sites off their cell's last
// column and row, then sites on one of them, then the corners (BaseDTInnerDBSH::systemLoopDC,
// kpz/kpzSimulationPrimitivesTemplates_BaseInnerDB.cu:110-163).  Two attempts of a round touch a
// common bit only if one's site is the other's right or lower neighbour, and then the former
// lies in an earlier phase.  All attempts without such a neighbour commute, so they are done in
// one pass; the others (0.39 % of all, known from the positions alone) follow in their phases'
// order.  That takes one pass and on average 2.1 barriers a round (a block of 512 cells has two such
// attempts a round) instead of three of each.
// Columns, rows and word offsets of four rounds are formed as bytes of one word.  Measured on a
// B200, DBSH at p = 0.95, q = 0.05: 16384^2 1592 -> 1248 us per MCS, 1024^2 181 -> 156 us (a launch
// there is 8 blocks, 64 rounds one after the other); DBSHRep 1583 -> 1239, DTDBSH 929 -> 779 us at
// 16384^2.  The integer ALU bounds it.
//
// WARPS warps share a block; each owns DT_CY / WARPS cell rows, a cell column per lane, and loads a
// round's attempts of its rows together.
template <bool COUNT, bool DIS, int SCHEME, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, WARPS >= 16 ? 2 : 4)
dt_scatter_kernel(uint32_t* __restrict__ sys, int lxw, int lyw, int lnbx, int ox, int oy, int d, uint32_t t, const DtKey key,
                  uint32_t stream, Thresh tp, Thresh tq, unsigned long long* __restrict__ counters,
                  const uint32_t* __restrict__ dis, DisorderRates dr)
{
    constexpr bool REP = SCHEME == DT_SCHEME_DBSHREP;
    constexpr bool BORDER = SCHEME == DT_SCHEME_DBSH || SCHEME == DT_SCHEME_DB || REP;
    constexpr int ROWS = DT_CY / WARPS;  // cell rows of a warp
    constexpr int NT = 32 * WARPS;
    __shared__ uint32_t plane[(DIS ? 4 : 2) * PL_WORDS];
    __shared__ uint32_t hits_s[REP ? WARPS : 1];
    __shared__ uint32_t need_s[3];
    // rate classes: {whether a deposition (desorption) candidate can flip, its acceptance limit}; as
    // a kernel parameter indexed by lane the thresholds went through local memory (DBSH, four classes
    // with counters at 8192^2: 635 -> 444 us a MCS; two classes at 16384^2: 1651 -> 1383)
    __shared__ uint2 rate_s[DIS ? 8 : 1];
    const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t Wx = 1u << lxw, Wy = 1u << lyw;
    const uint32_t ax = ox & 3, ay = oy & 3;
    bool need_u = !(tp.always || tp.planes == 0) || !(tq.always || tq.planes == 0);
    if (DIS) need_u = dr.planes > 0;
    const DtRule rule = make_rule(tp, tq);
    unsigned long long ndep = 0, ndes = 0;

    const int b = (int)blockIdx.x;
    const uint32_t bx = b & ((1 << lnbx) - 1), by = b >> lnbx;
    const uint32_t wx0 = ((uint32_t)ox + (2 * bx + (d & 1)) * DT_BX) >> 2;
    const uint32_t wy0 = ((uint32_t)oy + (2 * by + (d >> 1)) * DT_BY) >> 2;
    planes_load(sys, plane, tid, NT, wx0, wy0, Wx, Wy);
    if (DIS) planes_load(dis, plane + 2 * PL_WORDS, tid, NT, wx0, wy0, Wx, Wy);
    if (tid < 3) need_s[tid] = 0u;
    if (DIS && tid == 0) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const DtRule r = make_rule(dr.tp[c], dr.tq[c]);
            rate_s[2 * c] = make_uint2(r.ok_p, r.lim_p);
            rate_s[2 * c + 1] = make_uint2(r.ok_q, r.lim_q);
        }
    }
    __syncthreads();

    const int row0 = warp * ROWS;
    const uint32_t cid0 = (uint32_t)b * DT_CELLS + (uint32_t)(32 * row0 + lane);
    const uint32_t cx = 8u * (uint32_t)lane, cy = 8u * (uint32_t)row0;
    auto draw = [&](uint32_t index, uint32_t tag, uint32_t n) {
        return philox_dt(make_uint4(index, t, (tag << 24) | ((uint32_t)d << 16) | n, stream), key);
    };
    auto next = [](uint4& v) {
        const uint32_t w = v.x;
        v.x = v.y;
        v.y = v.z;
        v.z = v.w;
        return w;
    };

    if (BORDER) {
        // Four rounds of the dead-border schemes.  pos: positions, a byte per round, of the warp's
        // cell rows and of the row below them; act: rounds a cell takes part in (a bit each); ob4: the
        // block-wide cell offset, a byte per round; need: which rounds have attempts that must wait for
        // a neighbour (bit j) and corners among them (bit 4 + j), over the block.
        auto four_rounds = [&](const uint32_t pos[ROWS + 1], const uint4 uu[ROWS], uint32_t ob4, int nrounds,
                               const uint32_t act[ROWS], bool skip_border, uint32_t* need) {
            if (SCHEME == DT_SCHEME_DB) ob4 = 0u;
            const uint32_t sx = (ob4 & 0x07070707u) + bytes4(ax), sy = ((ob4 >> 3) & 0x07070707u) + bytes4(ay);
            uint32_t xb[ROWS], yb[ROWS], wb[ROWS];  // column, row and word offset of each round's site
            uint32_t go[ROWS], late[ROWS];          // bit 8 j + 7: attempted at once, or after its neighbour
            uint32_t mine = 0;
#pragma unroll
            for (int i = 0; i < ROWS; ++i) {
                const uint32_t p = pos[i];
                xb[i] = add_bytes(bytes4(cx), (p & 0x07070707u) + sx);
                yb[i] = (bytes4(cy + 8u * i) + ((p >> 3) & 0x07070707u) + sy) & 0x7F7F7F7Fu;
                wb[i] = (xb[i] >> 3) & 0x1C1C1C1Cu;
                const uint32_t in = act[i];
                if (skip_border) {
                    // off the border: neither offset is 7
                    const uint32_t bx = (p & 0x07070707u) + 0x01010101u, by = ((p >> 3) & 0x07070707u) + 0x01010101u;
                    go[i] = ~((bx | by) << 4) & 0x80808080u;
                    late[i] = 0u;
                } else {
                    const uint32_t apart = not_adjacent(p, __shfl_sync(0xffffffffu, p, (lane + 1) & 31), pos[i + 1]);
                    go[i] = apart & in;
                    late[i] = ~apart & in;
                    if (late[i]) {
                        const uint32_t c = ((p & 0x3F3F3F3Fu) + 0x01010101u) << 1;  // corner: px = py = 7
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            if ((late[i] >> (8 * j + 7)) & 1u) mine |= (((c >> (8 * j + 7)) & 1u) ? 0x11u : 0x01u) << j;
                        }
                    }
                }
            }
            if (!skip_border) {
                mine = __reduce_or_sync(0xffffffffu, mine);
                if (lane == 0 && mine) atomicOr(need, mine);
            }
            uint32_t waits = 0;
            auto site = [&](int i, int j, DtSite<DIS>& s) {
                s.load(plane, xb[i] >> (8 * j), __byte_perm(yb[i], 0u, 0x4440 | j) * (4 * PL_W) + __byte_perm(wb[i], 0u, 0x4440 | j));
            };
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j >= nrounds) break;
                DtSite<DIS> s[ROWS];
#pragma unroll
                for (int i = 0; i < ROWS; ++i)
                    if ((go[i] >> (8 * j + 7)) & 1u) site(i, j, s[i]);
#pragma unroll
                for (int i = 0; i < ROWS; ++i)
                    if ((go[i] >> (8 * j + 7)) & 1u) s[i].template flip<COUNT>(pick4(uu[i], j), rule, rate_s, ndep, ndes);
                __syncthreads();
                if (skip_border) continue;
                if (j == 0) waits = *need;
#pragma unroll 1
                for (int phase = 1; phase <= 2; ++phase) {
                    if (!((waits >> (phase == 2 ? 4 + j : j)) & 1u)) break;
#pragma unroll
                    for (int i = 0; i < ROWS; ++i) {
                        const bool corner = ((pos[i] >> (8 * j)) & 0x3Fu) == 0x3Fu;
                        if (((late[i] >> (8 * j + 7)) & 1u) && corner == (phase == 2)) {
                            DtSite<DIS> s1;
                            site(i, j, s1);
                            s1.template flip<COUNT>(pick4(uu[i], j), rule, rate_s, ndep, ndes);
                        }
                    }
                    __syncthreads();
                }
            }
        };
        uint32_t hits = 0;
        uint32_t all[ROWS];
#pragma unroll
        for (int i = 0; i < ROWS; ++i) all[i] = 0x80808080u;
        uint4 ow, pw[ROWS + 1];
#pragma unroll 1
        for (int q = 0; q < DT_ROUNDS / 4; ++q) {
            if ((q & 3) == 0) {
                ow = draw((uint32_t)b, TAG_DBSH_ORIGIN, q >> 2);
#pragma unroll
                for (int i = 0; i <= ROWS; ++i) {
                    // the row below the warp's last (the cells' torus) only for its positions
                    const uint32_t c = i < ROWS ? cid0 + 32u * i
                                                : (uint32_t)b * DT_CELLS + (uint32_t)(32 * ((row0 + ROWS) & (DT_CY - 1)) + lane);
                    pw[i] = draw(c, TAG_DBSH_POS, q >> 2);
                }
            }
            uint32_t pos[ROWS + 1];
            uint4 uu[ROWS];
#pragma unroll
            for (int i = 0; i <= ROWS; ++i) pos[i] = next(pw[i]);
#pragma unroll
            for (int i = 0; i < ROWS; ++i) {
                uu[i] = need_u ? draw(cid0 + 32u * i, TAG_DT, q) : make_uint4(0u, 0u, 0u, 0u);
                if (REP) {
                    // BaseDTInnerDBSHRep (:175-268): a border hit is not done in its round but counted,
                    // and after the 64 rounds the block makes that many fresh attempts, 512 per
                    // repetition round, each again in the three phases
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t p = pos[i] >> (8 * j);
                        // the block's count as the reference's reduction forms it (:214-227): the hits of
                        // the first cell and of cell rows 1.. -- those of row 0's other cells are not
                        // repeated there, nor here
                        if (((p & 7u) == 7u || (p & 0x38u) == 0x38u) && (row0 + i > 0 || lane == 0)) ++hits;
                    }
                }
            }
            // the word used two batches ago: every thread has read it before this batch's first barrier
            if (!REP && tid == 0) need_s[(q + 1) % 3] = 0u;
            four_rounds(pos, uu, next(ow), 4, all, REP, &need_s[q % 3]);
        }
        if (REP) {
            hits = __reduce_add_sync(0xffffffffu, hits);
            if (lane == 0) hits_s[warp] = hits;
            __syncthreads();
            uint32_t total = 0;
            for (int w = 0; w < WARPS; ++w) total += hits_s[w];
            const int nk = (int)((total + DT_CELLS - 1) / DT_CELLS);
#pragma unroll 1
            for (int q = 0; 4 * q < nk; ++q) {
                if ((q & 3) == 0) {
                    ow = draw((uint32_t)b, TAG_REP_ORIGIN, q >> 2);
#pragma unroll
                    for (int i = 0; i <= ROWS; ++i) {
                        const uint32_t c = i < ROWS ? cid0 + 32u * i
                                                    : (uint32_t)b * DT_CELLS + (uint32_t)(32 * ((row0 + ROWS) & (DT_CY - 1)) + lane);
                        pw[i] = draw(c, TAG_REP_POS, q >> 2);
                    }
                }
                uint32_t pos[ROWS + 1], act[ROWS];
                uint4 uu[ROWS];
#pragma unroll
                for (int i = 0; i <= ROWS; ++i) pos[i] = next(pw[i]);
#pragma unroll
                for (int i = 0; i < ROWS; ++i) {
                    uu[i] = need_u ? draw(cid0 + 32u * i, TAG_REP_U, q) : make_uint4(0u, 0u, 0u, 0u);
                    act[i] = 0u;
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if ((uint32_t)(4 * q + j) * DT_CELLS + (uint32_t)(32 * (row0 + i) + lane) < total) act[i] |= 0x80u << (8 * j);
                }
                if (tid == 0) need_s[(q + 1) % 3] = 0u;
                four_rounds(pos, uu, next(ow), nk - 4 * q < 4 ? nk - 4 * q : 4, act, false, &need_s[q % 3]);
            }
        }
    } else {
        // BaseDTInnerDTDBSH (kpz/kpzSimulationPrimitivesTemplates_BaseInnerDTr.cu:30-85): a
        // quadrant of the cells and a block-wide offset in [0,8)^2 per round, the site wrapped inside
        // the block before the origin's in-word offset is added; neighbouring cells' sites stay 4 or
        // more sites apart.  Quadrants (2 bits per round; every thread derives the same words) and
        // offsets of four rounds lie in the bytes of one word, as do the wrapped columns and rows.
        uint4 sub = draw((uint32_t)b, TAG_DT_SUB, 0u);
        uint4 ow = make_uint4(0u, 0u, 0u, 0u), pw[ROWS];
        uint32_t sw = 0, pos[ROWS];
        uint32_t* const first = plane + ay * PL_W;
#pragma unroll 1
        for (int q = 0; q < DT_ROUNDS / 4; ++q) {
            if ((q & 3) == 0) {
                sw = next(sub);
                ow = draw((uint32_t)b, TAG_DBSH_ORIGIN, q >> 2);
            }
            const uint32_t ob4 = next(ow);
            uint32_t sc4 = sw & 0xFFu;
            sw >>= 8;
            sc4 = (sc4 | (sc4 << 12)) & 0x000F000Fu;
            sc4 = (sc4 | (sc4 << 6)) & 0x03030303u;
            const uint32_t sx = ((sc4 & 0x01010101u) << 2) + (ob4 & 0x07070707u);
            const uint32_t sy = ((sc4 & 0x02020202u) << 1) + ((ob4 >> 3) & 0x07070707u);
            uint4 uu[ROWS];
            uint32_t xb[ROWS], yb[ROWS];
#pragma unroll
            for (int i = 0; i < ROWS; ++i) {
                if ((q & 7) == 0) pw[i] = draw(cid0 + 32u * i, TAG_DT_POS, q >> 3);
                pos[i] = (q & 1) ? pos[i] >> 16 : next(pw[i]);
                uu[i] = need_u ? draw(cid0 + 32u * i, TAG_DT, q) : make_uint4(0u, 0u, 0u, 0u);
                // positions of four rounds, a nibble each (x in bits 0-1, y in bits 2-3), to bytes
                uint32_t p = __byte_perm(pos[i], 0u, 0x4140);
                p = (p | (p << 4)) & 0x0F0F0F0Fu;
                xb[i] = add_bytes(bytes4(cx), (p & 0x03030303u) + sx);
                yb[i] = (bytes4(cy + 8u * i) + (p >> 2 & 0x03030303u) + sy) & 0x7F7F7F7Fu;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                DtSite<DIS> s[ROWS];
#pragma unroll
                for (int i = 0; i < ROWS; ++i) {
                    const uint32_t x = __byte_perm(xb[i], 0u, 0x4440 | j) + ax;
                    s[i].load(first, x, __byte_perm(yb[i], 0u, 0x4440 | j) * (4 * PL_W) + ((x >> 3) & 0x7Cu));
                }
#pragma unroll
                for (int i = 0; i < ROWS; ++i) s[i].template flip<COUNT>(pick4(uu[i], j), rule, rate_s, ndep, ndes);
                __syncthreads();
            }
        }
    }
    planes_store(sys, plane, tid, NT, wx0, wy0, Wx, Wy);
    if (COUNT) {
        for (int o = 16; o > 0; o >>= 1) {
            ndep += __shfl_xor_sync(0xffffffffu, ndep, o);
            ndes += __shfl_xor_sync(0xffffffffu, ndes, o);
        }
        if (lane == 0 && (ndep | ndes)) {
            atomicAdd(&counters[0], ndep);
            atomicAdd(&counters[1], ndes);
        }
    }
}

// ---- DT and DB4: one quadrant of every cell per round ----
//
// 32 x 16 threads, one cell each, on the block's ENC_LOCAL words in shared memory (65 x 33 with the
// halo).  No two sites of a round share a word, so a round needs one barrier and its flips only
// order themselves.  A per-launch table of 8-byte entries turns (quadrant, position) into the three
// words' byte offsets and three rotate amounts.  59 instructions an attempt, most of them on the
// integer ALU (2 cycles each per warp and scheduler), which bounds it.  Holding the cells in
// registers instead (quadrant and neighbours by shifts and shuffles, no tile and no barrier in most
// rounds) took 63 and was 2 % faster at 16384^2 and 10 % slower below 4096^2, and was dropped.
constexpr int DT_TX = 32, DT_TY = 16;
constexpr int DT_THREADS = DT_TX * DT_TY;
constexpr int DT_TW = DT_BXW + 1, DT_TH = DT_BYW + 1;  // shared tile with halo
// DB4: sites of a block whose x >= 251 or y >= 123 (before the origin's offset inside a word)
// are dead, so no update reaches past the block (LocalLayoutDB4::BLOCK_BORDER_WIDTH = 5,
// kpz/LocalLayout.h:120-131)
constexpr int DB4_BORDER = 5;

// Site-table entry of the site (vx, vy) sites right of and below a word (a thread cell's first
// word, or the tile's): the tile words of the site, its right neighbour and its lower neighbour
// relative to that word, and the rotate amounts
//   bits 0-7: the site's shift sh (its two slope bits rotate down to bits 0-1),
//   8-15: (shr - 2) mod 32 (the right neighbour's x-slope bit rotates to bit 2),
//   16-23: (shd - 3) mod 32 (the lower neighbour's y-slope bit rotates to bit 3);
// a funnel shift uses its amount modulo 32, so no field needs a mask.
__device__ __forceinline__ uint4 site_entry(int vx, int vy)
{
    const uint32_t sh = (uint32_t)(((vx & 3) << 1) | ((vy & 3) << 3));
    const uint32_t shr = (uint32_t)((((vx + 1) & 3) << 1) | ((vy & 3) << 3));
    const uint32_t shd = (uint32_t)(((vx & 3) << 1) | (((vy + 1) & 3) << 3) | 1);
    return make_uint4((uint32_t)((vy >> 2) * DT_TW + (vx >> 2)), (uint32_t)((vy >> 2) * DT_TW + ((vx + 1) >> 2)),
                      (uint32_t)(((vy + 1) >> 2) * DT_TW + (vx >> 2)),
                      sh | (((shr - 2u) & 31u) << 8) | (((shd - 3u) & 31u) << 16));
}
// An 8-byte table entry in shared memory, with byte offsets so that an address is one add to
// a byte base: x = 4 w | 4 w_right << 16, y = 4 w_down | sh << 11 | (shr - 2) << 16 |
// (shd - 3) << 21 (the rotate amounts of site_entry, each read by shifting y right and used
// modulo 32); bits 26-27 are left for flags.
__device__ __forceinline__ uint2 pack_entry_bytes(const uint4 e)
{
    return make_uint2((4u * e.x) | ((4u * e.y) << 16),
                      (4u * e.z) | ((e.w & 31u) << 11) | (((e.w >> 8) & 31u) << 16) | (((e.w >> 16) & 31u) << 21));
}

template <bool COUNT, bool DIS, int SCHEME>
__global__ void __launch_bounds__(DT_THREADS, 4)
dt_quadrant_kernel(uint32_t* __restrict__ sys, int lxw, int lyw, int lnbx, int nblocks, int ox, int oy,
          int d, uint32_t t, const DtKey key, uint32_t stream, Thresh tp, Thresh tq,
          unsigned long long* __restrict__ counters, const uint32_t* __restrict__ dis, DisorderRates dr)
{
    constexpr bool DB4 = SCHEME == DT_SCHEME_DB4;
    // a 64-entry table by (quadrant, position): the origin's offset inside a word (ox & 3, oy & 3) is
    // the launch's, so it is folded in
    constexpr int NLUT = 64;
    constexpr int ROUNDS = DB4 ? DT_ROUNDS / 2 : DT_ROUNDS;
    constexpr uint32_t T_SUB = DB4 ? TAG_DB4_SUB : TAG_DT_SUB;
    constexpr uint32_t T_POS = DB4 ? TAG_DB4_POS : TAG_DT_POS;
    constexpr uint32_t T_U = DB4 ? TAG_DB4_U : TAG_DT;
    __shared__ uint32_t tile[DT_TH * DT_TW];
    __shared__ uint32_t dtile[DIS ? DT_TH * DT_TW : 1];
    __shared__ uint2 lut[NLUT];
    const int tid = threadIdx.y * DT_TX + threadIdx.x;
    const uint32_t Wx = 1u << lxw, Wy = 1u << lyw;
    const int ax = ox & 3, ay = oy & 3;
    bool need_u = !(tp.always || tp.planes == 0) || !(tq.always || tq.planes == 0);
    if (DIS) need_u = dr.planes > 0;
    // the rule's candidates and acceptance limits: a site with configuration cfg_p (12, or an
    // impossible 16 when p = 0) flips when u <= lim_p = T_p - 1; likewise q (configuration 3)
    const uint32_t cfg_p = (tp.always || tp.planes) ? 12u : 16u, cfg_q = (tq.always || tq.planes) ? 3u : 16u;
    const uint32_t lim_p = tp.always ? 0xFFFFFFFFu : tp.t - 1u, lim_q = tq.always ? 0xFFFFFFFFu : tq.t - 1u;
    unsigned long long ndep = 0, ndes = 0;
    {
        if (tid < NLUT) {
            // bits 25 / 26 of y: the site lies at in-cell x / y >= 3, DB4's dead border when the cell
            // is the block's last in its row / column (it starts 8 sites before the block's edge)
            const int sc = tid >> 4, pb = tid & 15;
            const int ux = 4 * (sc & 1) + (pb & 3), uy = 4 * (sc >> 1) + (pb >> 2);
            uint2 e = pack_entry_bytes(site_entry(ux + ax, uy + ay));
            e.y |= (ux >= 8 - DB4_BORDER ? 1u << 26 : 0u) | (uy >= 8 - DB4_BORDER ? 1u << 27 : 0u);
            lut[tid] = e;
        }
    }
    // DB4: the last thread column / row owns the block's dead border
    const uint32_t dead_mask = (threadIdx.x == DT_TX - 1 ? 1u << 26 : 0u) | (threadIdx.y == DT_TY - 1 ? 1u << 27 : 0u);
    const int tbase = 2 * threadIdx.y * DT_TW + 2 * threadIdx.x;
    // the thread cell's first word in the tiles, as byte pointers for the DT / DB4 table
    char* tcell = reinterpret_cast<char*>(tile + tbase);
    const char* dcell = reinterpret_cast<const char*>(dtile + (DIS ? tbase : 0));
    for (int b = blockIdx.x; b < nblocks; b += gridDim.x) {
        const int bx = b & ((1 << lnbx) - 1), by = b >> lnbx;
        const uint32_t X0 = (uint32_t)ox + (uint32_t)(DB4 ? bx : 2 * bx + (d & 1)) * DT_BX;
        const uint32_t Y0 = (uint32_t)oy + (uint32_t)(DB4 ? by : 2 * by + (d >> 1)) * DT_BY;
        const uint32_t wx0 = X0 >> 2, wy0 = Y0 >> 2;
        for (int i = tid; i < DT_TH * DT_TW; i += DT_THREADS) {
            const uint32_t r = i / DT_TW, c = i - r * DT_TW;
            // DB4 blocks tile the lattice without halo: the dead border keeps every update,
            // its right and its lower neighbour inside the block's 64x32 words
            if (DB4 && (r == DT_BYW || c == DT_BXW)) continue;
            const size_t gi = (size_t)((wy0 + r) & (Wy - 1)) * Wx + ((wx0 + c) & (Wx - 1));
            tile[i] = sys[gi];
            if (DIS) dtile[i] = dis[gi];
        }
        // block-wide sub-cell sequence: 2 bits per round (every thread derives the same words)
        const uint4 sub = philox_dt(
            make_uint4((uint32_t)b, t, (T_SUB << 24) | ((uint32_t)d << 16), stream), key);
        const uint32_t cid = (uint32_t)b * DT_THREADS + (uint32_t)tid;
        __syncthreads();
        uint4 pos = make_uint4(0, 0, 0, 0), uu = make_uint4(0, 0, 0, 0);
        // all rounds unrolled: four batches at a time the plain instance spilled 24 bytes and the counting
        // one 40 under the 32 registers of four CTAs per SM (16384^2, p = 1, q = 0: 559 us a MCS,
        // counting 627; now 532 and 591; at p = 0.95, q = 0.05: 720 -> 682)
#pragma unroll
        for (int rb = 0; rb < ROUNDS; rb += 8) {
            if ((rb & 31) == 0)
                pos = philox_dt(
                    make_uint4(cid, t, (T_POS << 24) | ((uint32_t)d << 16) | (uint32_t)(rb >> 5), stream), key);
            const uint32_t sw = pick4(sub, rb >> 4);
            const uint32_t pw = pick4(pos, (rb & 31) >> 3);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int r = rb + j;
                if (need_u && (j & 3) == 0)
                    uu = philox_dt(
                        make_uint4(cid, t, (T_U << 24) | ((uint32_t)d << 16) | (uint32_t)(r >> 2), stream), key);
                const uint32_t sc = (sw >> (2 * (r & 15))) & 3u;
                const uint32_t pb = (pw >> (4 * j)) & 15u;
                const uint32_t u = pick4(uu, j & 3);
                {
                    const uint2 e = lut[sc * 16u + pb];
                    if (!DB4 || (e.y & dead_mask) == 0u) {
                        uint32_t* pw = reinterpret_cast<uint32_t*>(tcell + (e.x & 0xFFFFu));
                        uint32_t* pr = reinterpret_cast<uint32_t*>(tcell + (e.x >> 16));
                        uint32_t* pd = reinterpret_cast<uint32_t*>(tcell + (e.y & 2047u));
                        const uint32_t r1 = e.y >> 11, r2 = e.y >> 16, r3 = e.y >> 21;
                        const uint32_t cw = *pw, rw = *pr, dw = *pd;
                        const uint32_t cfg = (__funnelshift_r(cw, cw, r1) & 3u) | (__funnelshift_r(rw, rw, r2) & 4u) |
                                             (__funnelshift_r(dw, dw, r3) & 8u);
                        bool flip, is_p;
                        if (DIS) {
                            is_p = cfg == 12u;
                            flip = false;
                            if (is_p || cfg == 3u) {
                                const uint32_t dw0 = *reinterpret_cast<const uint32_t*>(dcell + (e.x & 0xFFFFu));
                                const int cls = (int)(__funnelshift_r(dw0, dw0, r1) & 3u);
                                const Thresh& th = is_p ? dr.tp[cls] : dr.tq[cls];
                                flip = th.always || (th.planes && u < th.t);
                            }
                        } else {
                            is_p = cfg == cfg_p;
                            flip = (is_p || cfg == cfg_q) && u <= (is_p ? lim_p : lim_q);
                        }
                        if (flip) {
                            atomicXor(pw, __funnelshift_l(3u, 3u, r1));
                            atomicXor(pr, __funnelshift_l(4u, 4u, r2));
                            atomicXor(pd, __funnelshift_l(8u, 8u, r3));
                            if (COUNT) {
                                if (is_p) ++ndep;
                                else ++ndes;
                            }
                        }
                    }
                }
                __syncthreads();
            }
        }
        for (int i = tid; i < DT_TH * DT_TW; i += DT_THREADS) {
            const uint32_t r = i / DT_TW, c = i - r * DT_TW;
            if (DB4 && (r == DT_BYW || c == DT_BXW)) continue;
            sys[(size_t)((wy0 + r) & (Wy - 1)) * Wx + ((wx0 + c) & (Wx - 1))] = tile[i];
        }
        __syncthreads();
    }
    if (COUNT) {
        for (int o = 16; o > 0; o >>= 1) {
            ndep += __shfl_xor_sync(0xffffffffu, ndep, o);
            ndes += __shfl_xor_sync(0xffffffffu, ndes, o);
        }
        if ((tid & 31) == 0 && (ndep | ndes)) {
            atomicAdd(&counters[0], ndep);
            atomicAdd(&counters[1], ndes);
        }
    }
}

// Warps of a scattered-site block: eight (two cell rows each) where the blocks fill the SMs, else
// sixteen, whose rounds are shortest.  DBSH at 16384^2 (2048 blocks a launch): 8 warps 1247 us per
// MCS, 16 warps 1420, 4 warps 1311; at 8192^2 (512): 8 warps 397, 16 warps 432; at 8192 x 4096 (256):
// 16 warps 232, 8 warps 250; at 4096^2 (128): 16 warps 158 us, 8 warps 197.  DTDBSH at 256 blocks: 150
// either way.
constexpr int DT_WARPS_MANY = 8, DT_WARPS_FEW = 16;

// Host copy of the Philox4x32-10 bijection for the per-MCS origin and domain-set order (and
// the random measurement spacing of kpzb_sample_times).
void philox_host(const uint32_t ctr[4], uint64_t seed, uint32_t out[4])
{
    uint32_t c0 = ctr[0], c1 = ctr[1], c2 = ctr[2], c3 = ctr[3];
    uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
    for (int r = 0; r < 10; ++r) {
        if (r) {
            k0 += 0x9E3779B9u;
            k1 += 0xBB67AE85u;
        }
        const uint64_t p0 = (uint64_t)0xD2511F53u * c0, p1 = (uint64_t)0xCD9E8D57u * c2;
        const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c1 ^ k0, n2 = (uint32_t)(p0 >> 32) ^ c3 ^ k1;
        c0 = n0;
        c1 = (uint32_t)p1;
        c2 = n2;
        c3 = (uint32_t)p0;
    }
    out[0] = c0;
    out[1] = c1;
    out[2] = c2;
    out[3] = c3;
}

// Origin in [0, 2*block) sites and the Kmc::Shuffle<4> order (inc/shuffle.h:76-90).
static void dt_plan(uint64_t seed, uint32_t stream, uint32_t t, int* ox, int* oy, int order[4])
{
    const uint32_t ctr[4] = {0u, t, TAG_DT_ORIGIN << 24, stream};
    uint32_t r[4];
    philox_host(ctr, seed, r);
    *ox = (int)(r[0] & (uint32_t)(2 * DT_BX - 1));
    *oy = (int)(r[1] & (uint32_t)(2 * DT_BY - 1));
    uint32_t rnd = r[2];
    for (int a = 0; a < 4; ++a) order[a] = a;
    for (int a = 0; a < 4; ++a) {
        const int i = (int)(rnd & 3u);
        const int v = order[i];
        order[i] = order[a];
        order[a] = v;
        rnd >>= 2;
    }
}

kpzb_status dt_init(DtState* s, int lx, int ly, int sm_count, bool db4)
{
    if (db4 && (lx < 8 || ly < 7)) return fail(KPZB_EINVAL, "DB4 needs lx >= 8 and ly >= 7 (one 256x128 block)");
    if (!db4 && (lx < 9 || ly < 8))
        return fail(KPZB_EINVAL, "DT needs lx >= 9 and ly >= 8 (one 512x256 double tile)");
    s->sm_count = sm_count;
    if (db4) s->scheme = DT_SCHEME_DB4;
    s->ready = true;
    return KPZB_OK;
}

void dt_free(DtState* s) { s->ready = false; }

static uint64_t thresh_dt(double p)
{
    if (!(p > 0.0)) return 0;
    if (p >= 1.0) return 1ull << 32;
    const double t = std::ceil(p * 4294967296.0);
    return t >= 4294967296.0 ? (1ull << 32) : (uint64_t)t;
}

kpzb_status dt_enqueue(DtState* s, uint32_t* d_local, int lx, int ly, uint64_t t0, int n, double p,
                       double q, uint64_t seed, uint32_t stream, cudaStream_t st,
                       unsigned long long* d_counters, const uint32_t* dis, const uint64_t* dis_Tp,
                       const uint64_t* dis_Tq)
{
    if (!s->ready) return fail(KPZB_ESTATE, "DT state not initialised");
    const DtKey key = make_dt_key(make_key(seed));
    const Thresh tp = make_thresh(thresh_dt(p)), tq = make_thresh(thresh_dt(q));
    const bool db4 = s->scheme == DT_SCHEME_DB4;
    const int lnbx = db4 ? lx - 8 : lx - 9;
    const int nblocks = (1 << lnbx) * (1 << (db4 ? ly - 7 : ly - 8));
    const DisorderRates dr = dis ? make_disorder_rates(dis_Tp, dis_Tq) : DisorderRates{};
    const bool c = d_counters != nullptr, ds = dis != nullptr;
    const bool few = nblocks <= 2 * s->sm_count;
    auto launch = [&](int ox, int oy, int d, uint32_t t) {
        if (s->scheme == DT_SCHEME_DT || db4) {
            const int grid = nblocks < 4 * s->sm_count ? nblocks : 4 * s->sm_count;
            auto go = [&](auto kern) {
                kern<<<grid, dim3(DT_TX, DT_TY), 0, st>>>(d_local, lx - 2, ly - 2, lnbx, nblocks, ox, oy, d, t, key,
                                                          stream, tp, tq, d_counters, dis, dr);
            };
            if (db4) c ? go(dt_quadrant_kernel<true, false, DT_SCHEME_DB4>) : go(dt_quadrant_kernel<false, false, DT_SCHEME_DB4>);
            else if (c && ds) go(dt_quadrant_kernel<true, true, DT_SCHEME_DT>);
            else if (c) go(dt_quadrant_kernel<true, false, DT_SCHEME_DT>);
            else if (ds) go(dt_quadrant_kernel<false, true, DT_SCHEME_DT>);
            else go(dt_quadrant_kernel<false, false, DT_SCHEME_DT>);
            return;
        }
        auto pick = [&](auto scheme_tag, auto warps_tag) {
            constexpr int S = decltype(scheme_tag)::value, W = decltype(warps_tag)::value;
            auto go = [&](auto kern) {
                kern<<<nblocks, 32 * W, 0, st>>>(d_local, lx - 2, ly - 2, lnbx, ox, oy, d, t, key, stream, tp, tq,
                                                 d_counters, dis, dr);
            };
            if (c && ds) go(dt_scatter_kernel<true, true, S, W>);
            else if (c) go(dt_scatter_kernel<true, false, S, W>);
            else if (ds) go(dt_scatter_kernel<false, true, S, W>);
            else go(dt_scatter_kernel<false, false, S, W>);
        };
        auto size = [&](auto scheme_tag) {
            if (few) pick(scheme_tag, std::integral_constant<int, DT_WARPS_FEW>{});
            else pick(scheme_tag, std::integral_constant<int, DT_WARPS_MANY>{});
        };
        switch (s->scheme) {
        case DT_SCHEME_DBSH: size(std::integral_constant<int, DT_SCHEME_DBSH>{}); break;
        case DT_SCHEME_DB: size(std::integral_constant<int, DT_SCHEME_DB>{}); break;
        case DT_SCHEME_DBSHREP: size(std::integral_constant<int, DT_SCHEME_DBSHREP>{}); break;
        default: size(std::integral_constant<int, DT_SCHEME_DTDBSH>{}); break;
        }
    };
    for (int i = 0; i < n; ++i) {
        const uint32_t t = (uint32_t)(t0 + (uint64_t)i);
        if (db4) {
            // Scheduler::doMcs (kpz/scheduler.cu:37-52): 2^L_MCS_DIV = 2 launches per MCS, each
            // over every block from a random origin in [0, block) sites
            for (int a = 0; a < 2; ++a) {
                const uint32_t ctr[4] = {(uint32_t)a, t, TAG_DB4_ORIGIN << 24, stream};
                uint32_t r[4];
                philox_host(ctr, seed, r);
                launch((int)(r[0] & (uint32_t)(DT_BX - 1)), (int)(r[1] & (uint32_t)(DT_BY - 1)), a, t);
            }
        } else {
            int ox, oy, order[4];
            dt_plan(seed, stream, t, &ox, &oy, order);
            for (int a = 0; a < 4; ++a) launch(ox, oy, order[a], t);
        }
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return cuda_fail(e, "DT launch");
    }
    return KPZB_OK;
}

}  // namespace kpzb
