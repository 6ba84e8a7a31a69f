// kpzb_common.cuh -- device helpers shared by the kpzb kernels (sm_100a).
//
// Counter-based random stream (the one the CPU oracle restates):
//   Philox4x32-10 (Salmon et al., SC'11), key = (seed lo, seed hi),
//   counter = (qword >> 2, step, plane | tag << 8, stream); output word qword & 3.
//   qword: word index inside an ENC_CBBIT quadrant; step = 2*t + sublattice;
//   plane k supplies bit (31-k) of each site's 32-bit uniform u.
// Decision: local minimum flips iff u < T(p), local maximum iff u < T(q),
//   T(x) = min(2^32, ceil(x * 2^32)).  Evaluated bit-serially from the MSB
//   plane, 32 sites per word at once, stopping when no site is undecided.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace kpzb {

constexpr uint32_t TAG_SCA = 1u;
constexpr uint32_t TAG_DT = 2u;
constexpr uint32_t TAG_DT_ORIGIN = 3u;

struct Key {
    uint32_t k0, k1;
};

__host__ __device__ __forceinline__ Key make_key(uint64_t seed)
{
    return Key{(uint32_t)seed, (uint32_t)(seed >> 32)};
}

// Philox4x32-10 round function and Weyl key schedule (SC'11, sec. 3.2).
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, Key k)
{
    uint32_t k0 = k.k0, k1 = k.k1;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        if (r) {
            k0 += 0x9E3779B9u;
            k1 += 0xBB67AE85u;
        }
        const uint32_t lo0 = 0xD2511F53u * c.x;
        const uint32_t hi0 = __umulhi(0xD2511F53u, c.x);
        const uint32_t lo1 = 0xCD9E8D57u * c.z;
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z);
        c = make_uint4(hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0);
    }
    return c;
}

// Threshold as (flag, low 32 bits): always = T >= 2^32; never = T == 0;
// planes = number of MSB planes that can decide (32 - ctz(T)).
struct Thresh {
    uint32_t t;      // low 32 bits of T (T < 2^32 when !always)
    int planes;      // 0 when always or never
    bool always;
};

__host__ __device__ inline Thresh make_thresh(uint64_t T)
{
    Thresh r;
    r.always = T >= (1ull << 32);
    r.t = r.always ? 0u : (uint32_t)T;
    int planes = 0;
    if (!r.always && r.t) {
        uint32_t v = r.t;
        int ctz = 0;
        while (!(v & 1u)) {
            v >>= 1;
            ++ctz;
        }
        planes = 32 - ctz;
    }
    r.planes = planes;
    return r;
}

// The first two Philox rounds of a decision's planes, split into what depends on the site group
// and what depends on the plane.  The planes of one group and half-step share counter words 0, 1
// and 3 and differ in word 2 alone, so round 1 multiplies the group index and the plane
// separately, and in round 2 the product with counter word 0 depends only on the plane and the
// one with word 2 only on the group: the state after round 2 is
//   { g.a ^ p.x, g.b, g.c ^ p.z, p.w }
// and a plane costs eight rounds instead of ten.  A round's two 32 x 32 -> 64 bit products take 4.25
// cycles each per warp and scheduler, twice a logic operation, so rounds are what a plane is
// made of.  With the comparison below: (0.95,0.05) at 8192^2 49 -> 42 us per MCS, binary disorder at
// 4096 x 2048 20 -> 15.6 us.
struct PlanePart {
    uint32_t x, z, w;
};
struct GroupPart {
    uint32_t a, b, c;
};
__host__ __device__ __forceinline__ PlanePart plane_part(uint32_t plane, uint32_t step, Key k)
{
    const uint64_t p1 = (uint64_t)0xCD9E8D57u * (plane | (TAG_SCA << 8));
    const uint64_t p0 = (uint64_t)0xD2511F53u * ((uint32_t)(p1 >> 32) ^ step ^ k.k0);
    return PlanePart{(uint32_t)p1 ^ (k.k0 + 0x9E3779B9u), (uint32_t)(p0 >> 32) ^ (k.k1 + 0xBB67AE85u), (uint32_t)p0};
}
__device__ __forceinline__ GroupPart group_part(uint32_t qgroup, uint32_t stream, Key k)
{
    const uint64_t p0 = (uint64_t)0xD2511F53u * qgroup;
    const uint64_t p1 = (uint64_t)0xCD9E8D57u * ((uint32_t)(p0 >> 32) ^ stream ^ k.k1);
    return GroupPart{(uint32_t)(p1 >> 32), (uint32_t)p1, (uint32_t)p0};
}
__device__ __forceinline__ uint4 philox_plane(const GroupPart& g, const PlanePart& p, Key k)
{
    uint4 c = make_uint4(g.a ^ p.x, g.b, g.c ^ p.z, p.w);
    uint32_t k0 = k.k0 + 0x9E3779B9u, k1 = k.k1 + 0xBB67AE85u;
#pragma unroll
    for (int r = 2; r < 10; ++r) {
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
        const uint64_t p0 = (uint64_t)0xD2511F53u * c.x, p1 = (uint64_t)0xCD9E8D57u * c.z;
        c = make_uint4((uint32_t)(p1 >> 32) ^ c.y ^ k0, (uint32_t)p1, (uint32_t)(p0 >> 32) ^ c.w ^ k1, (uint32_t)p0);
    }
    return c;
}

// Plane parts of one half-step: all 32 as a table (a kernel parameter), or made as they are needed.
struct PlaneTable {
    PlanePart p[32];
    __device__ __forceinline__ PlanePart at(int k) const { return p[k]; }
};
inline PlaneTable make_plane_table(uint32_t step, Key key)
{
    PlaneTable t;
    for (uint32_t k = 0; k < 32; ++k) t.p[k] = plane_part(k, step, key);
    return t;
}
struct PlaneMaker {
    uint32_t step;
    Key key;
    __device__ __forceinline__ PlanePart at(int k) const { return plane_part((uint32_t)k, step, key); }
};

// Bit-serial comparison of a group's 128 uniforms with their sites' thresholds: `eq` marks the
// sites whose u still equals the threshold's leading planes, `flip` the outcome of the others.  At
// each plane an undecided site takes its threshold's bit as its outcome; it is decided there when
// its own bit differs (1 against 0: u < T), and its outcome then stands.  Three logic operations a
// word and plane (with separate masks for the two kinds of candidate and their decided flips it was
// six, and selecting each kind's bits two more).  Planes are fetched while a site is undecided,
// the first four -- a group has about 64 candidates -- without asking.  TB: threshold bit words
// of plane k; DROP: sites whose threshold has no 1 bit left below plane k (u < T is then false).
// WARP: all 32 lanes call together, with sixteen bytes of shared memory per warp in `slot`.  A warp
// runs until its slowest lane is done, 12.6 planes at (0.95,0.05) where a lane needs 7.5; so once
// at most half (a quarter) of the lanes have sites left, two (four) lanes compute two (four) planes
// of each such group at a time: (0.95,0.05) 42 -> 38.5 us per MCS at 8192^2, 138 -> 121 at 16384^2.
template <bool WARP, class Planes, class TB, class DROP>
__device__ __forceinline__ uint4 decide_planes(uint4 eq, uint4 flip, int kmax, Key key, const GroupPart& g,
                                               const Planes& planes, const TB& tb, const DROP& drop, uint8_t* slot)
{
    auto apply = [&](int k, const uint4& r) {
        const uint4 b = tb(k);
        flip.x = (eq.x & b.x) | (~eq.x & flip.x);
        flip.y = (eq.y & b.y) | (~eq.y & flip.y);
        flip.z = (eq.z & b.z) | (~eq.z & flip.z);
        flip.w = (eq.w & b.w) | (~eq.w & flip.w);
        eq.x &= ~(b.x ^ r.x);
        eq.y &= ~(b.y ^ r.y);
        eq.z &= ~(b.z ^ r.z);
        eq.w &= ~(b.w ^ r.w);
        drop(k, eq, flip);
    };
    auto plane = [&](int k) { apply(k, philox_plane(g, planes.at(k), key)); };
    int k = 0;
    if (kmax >= 4) {
#pragma unroll
        for (; k < 4; ++k) plane(k);
    }
    if (WARP && kmax > 4) {
        const int lane = (int)(threadIdx.x + threadIdx.y * blockDim.x) & 31;
        while (k < kmax) {
            const bool left = (eq.x | eq.y | eq.z | eq.w) != 0u;
            const uint32_t act = __ballot_sync(0xffffffffu, left);
            if (!act) break;
            const int n = __popc(act);
            if (n > 16) {
                plane(k++);
                continue;
            }
            const int lg = n > 8 ? 1 : 2, rank = __popc(act & ((1u << lane) - 1u));
            if (left) slot[rank] = (uint8_t)lane;
            __syncwarp();
            const int src = (int)slot[lane >> lg] & 31;  // entries past n: any lane, their planes go unused
            const GroupPart h{__shfl_sync(0xffffffffu, g.a, src), __shfl_sync(0xffffffffu, g.b, src),
                              __shfl_sync(0xffffffffu, g.c, src)};
            const uint4 r = philox_plane(h, planes.at(min(k + (lane & ((1 << lg) - 1)), 31)), key);
            __syncwarp();
            for (int j = 0; j < 1 << lg && k < kmax; ++j, ++k) {
                const int from = (rank << lg) + j;
                apply(k, make_uint4(__shfl_sync(0xffffffffu, r.x, from), __shfl_sync(0xffffffffu, r.y, from),
                                    __shfl_sync(0xffffffffu, r.z, from), __shfl_sync(0xffffffffu, r.w, from)));
            }
        }
    } else {
        for (; k < kmax && (eq.x | eq.y | eq.z | eq.w); ++k) plane(k);
    }
    // u equal to T in every plane: not below it
    return make_uint4(flip.x & ~eq.x, flip.y & ~eq.y, flip.z & ~eq.z, flip.w & ~eq.w);
}

// Four-word decision for the 128 sites of one Philox group (qgroup = qword >> 2).
// cp: local-minimum candidates, cq: local-maximum candidates. Returns the flip mask.
template <bool WARP = false, class Planes>
__device__ __forceinline__ uint4 decide4(uint4 cp, uint4 cq, Thresh tp, Thresh tq, Key key, uint32_t qgroup,
                                         const Planes& planes, uint32_t stream, uint8_t* slot = nullptr)
{
    const uint32_t ap = tp.always ? 0xFFFFFFFFu : 0u, aq = tq.always ? 0xFFFFFFFFu : 0u;
    const uint32_t hp = tp.planes ? 0xFFFFFFFFu : 0u, hq = tq.planes ? 0xFFFFFFFFu : 0u;
    const uint4 eq = make_uint4((cp.x & hp) | (cq.x & hq), (cp.y & hp) | (cq.y & hq), (cp.z & hp) | (cq.z & hq),
                                (cp.w & hp) | (cq.w & hq));
    const uint4 flip = make_uint4((cp.x & ap) | (cq.x & aq), (cp.y & ap) | (cq.y & aq), (cp.z & ap) | (cq.z & aq),
                                  (cp.w & ap) | (cq.w & aq));
    auto tb = [&](int k) {
        const uint32_t bp = (uint32_t)((int32_t)(tp.t << k) >> 31), bq = (uint32_t)((int32_t)(tq.t << k) >> 31);
        return make_uint4((cq.x & bq) | (~cq.x & bp), (cq.y & bq) | (~cq.y & bp), (cq.z & bq) | (~cq.z & bp),
                          (cq.w & bq) | (~cq.w & bp));
    };
    auto drop = [&](int k, uint4& e, uint4& f) {
        auto out = [&](uint32_t keep_p, uint32_t keep_q) {
            auto one = [&](uint32_t c, uint32_t& ew, uint32_t& fw) {
                const uint32_t keep = (c & keep_q) | (~c & keep_p);
                fw &= ~(ew & ~keep);
                ew &= keep;
            };
            one(cq.x, e.x, f.x);
            one(cq.y, e.y, f.y);
            one(cq.z, e.z, f.z);
            one(cq.w, e.w, f.w);
        };
        // (at the last plane of all, what is left is dropped anyway)
        if (k + 1 == tp.planes && tp.planes < tq.planes) out(0u, 0xFFFFFFFFu);
        if (k + 1 == tq.planes && tq.planes < tp.planes) out(0xFFFFFFFFu, 0u);
    };
    return decide_planes<WARP>(eq, flip, max(tp.planes, tq.planes), key, group_part(qgroup, stream, key), planes, tb,
                               drop, slot);
}

// The same decision for rates of at most three planes (DEC_FEW): whole Philox calls and a mask per
// kind of candidate.  With so few planes there is little to share and lanes hardly differ.  A 4-MCS
// band pass of 4096^2 at two CTAs per SM, this way against decide4: (0.75,0.25) 36.0 against 39.6
// us, (0.875,0.125) 45.6 against 48.7, but (0.9375,0.0625), four planes, 55.1 against 46.8.  The
// half-step kernel has its plane parts in a table and no instance of this: there decide4 is the
// faster one from two planes on ((0.75,0.25) at 4096^2 13.6 us a MCS against 14.6).
__device__ __forceinline__ uint4 decide4_few(uint4 cp, uint4 cq, Thresh tp, Thresh tq, Key key,
                                         uint32_t qgroup, uint32_t step, uint32_t stream)
{
    uint4 ltp, eqp, ltq, eqq;
    if (tp.always) {
        ltp = cp;
        eqp = make_uint4(0, 0, 0, 0);
    } else {
        ltp = make_uint4(0, 0, 0, 0);
        eqp = tp.planes ? cp : make_uint4(0, 0, 0, 0);
    }
    if (tq.always) {
        ltq = cq;
        eqq = make_uint4(0, 0, 0, 0);
    } else {
        ltq = make_uint4(0, 0, 0, 0);
        eqq = tq.planes ? cq : make_uint4(0, 0, 0, 0);
    }
    const int kmax = max(tp.planes, tq.planes);
    for (int k = 0; k < kmax; ++k) {
        const uint32_t any = eqp.x | eqp.y | eqp.z | eqp.w | eqq.x | eqq.y | eqq.z | eqq.w;
        if (!any) break;
        const uint4 r = philox4x32_10(make_uint4(qgroup, step, (uint32_t)k | (TAG_SCA << 8), stream), key);
        const uint32_t bp = (tp.t >> (31 - k)) & 1u;
        const uint32_t bq = (tq.t >> (31 - k)) & 1u;
        // bit of T is 1: sites with u-bit 0 are below T (decided), u-bit 1 stay equal.
        // bit of T is 0: sites with u-bit 1 are above T (drop), u-bit 0 stay equal.
        if (bp) {
            ltp.x |= eqp.x & ~r.x; ltp.y |= eqp.y & ~r.y; ltp.z |= eqp.z & ~r.z; ltp.w |= eqp.w & ~r.w;
            eqp.x &= r.x; eqp.y &= r.y; eqp.z &= r.z; eqp.w &= r.w;
        } else {
            eqp.x &= ~r.x; eqp.y &= ~r.y; eqp.z &= ~r.z; eqp.w &= ~r.w;
        }
        if (bq) {
            ltq.x |= eqq.x & ~r.x; ltq.y |= eqq.y & ~r.y; ltq.z |= eqq.z & ~r.z; ltq.w |= eqq.w & ~r.w;
            eqq.x &= r.x; eqq.y &= r.y; eqq.z &= r.z; eqq.w &= r.w;
        } else {
            eqq.x &= ~r.x; eqq.y &= ~r.y; eqq.z &= ~r.z; eqq.w &= ~r.w;
        }
        if (k + 1 >= tp.planes) eqp = make_uint4(0, 0, 0, 0);
        if (k + 1 >= tq.planes) eqq = make_uint4(0, 0, 0, 0);
    }
    return make_uint4(ltp.x | ltq.x, ltp.y | ltq.y, ltp.z | ltq.z, ltp.w | ltq.w);
}

// Decision modes, chosen once per launch from the two thresholds:
//   DEC_NONE   no random plane can matter (every threshold is 0 or 2^32),
//   DEC_ONE    at most the MSB plane matters (thresholds in {0, 2^31, 2^32}, e.g. p = 1/2),
//   DEC_GENERAL anything else (bit-serial loop of decide4).
//   DEC_FEW    DEC_GENERAL's rates of at most three planes, where a kernel has an instance of its own
//              for them (decide4_few).
// And for kernels whose rates are known only at run time, as in a batch:
//   DEC_ANY      any of these modes,
//   DEC_ANY_FEW  any of them but DEC_GENERAL.
enum DecMode { DEC_ANY_FEW = -2, DEC_ANY = -1, DEC_NONE = 0, DEC_ONE = 1, DEC_GENERAL = 2, DEC_FEW = 3 };

__host__ __device__ inline int dec_mode(Thresh tp, Thresh tq)
{
    const int m = tp.planes > tq.planes ? tp.planes : tq.planes;
    return m == 0 ? DEC_NONE : m == 1 ? DEC_ONE : DEC_GENERAL;
}

// The same with DEC_FEW told apart.
constexpr int DEC_FEW_PLANES = 3;
__host__ __device__ inline int dec_mode_few(Thresh tp, Thresh tq)
{
    const int m = dec_mode(tp, tq);
    return m == DEC_GENERAL && tp.planes <= DEC_FEW_PLANES && tq.planes <= DEC_FEW_PLANES ? (int)DEC_FEW : m;
}

// decide4 for at most one random plane (DEC_NONE, DEC_ONE); identical results.
__device__ __forceinline__ uint4 decide4_one(int mode, uint4 cp, uint4 cq, Thresh tp, Thresh tq, Key key,
                                             uint32_t qgroup, uint32_t step, uint32_t stream)
{
    if (mode == DEC_NONE) {
        const uint32_t ap = tp.always ? 0xFFFFFFFFu : 0u, aq = tq.always ? 0xFFFFFFFFu : 0u;
        return make_uint4((cp.x & ap) | (cq.x & aq), (cp.y & ap) | (cq.y & aq),
                          (cp.z & ap) | (cq.z & aq), (cp.w & ap) | (cq.w & aq));
    }
    // a threshold with one plane is 2^31: sites whose MSB of u is 0 flip
    const uint32_t any = cp.x | cp.y | cp.z | cp.w | cq.x | cq.y | cq.z | cq.w;
    uint4 r = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
    if (any) r = philox4x32_10(make_uint4(qgroup, step, TAG_SCA << 8, stream), key);
    const uint32_t ap = tp.always ? 0xFFFFFFFFu : 0u, aq = tq.always ? 0xFFFFFFFFu : 0u;
    const uint32_t hp = tp.planes ? 0xFFFFFFFFu : 0u, hq = tq.planes ? 0xFFFFFFFFu : 0u;
    return make_uint4((cp.x & (ap | (hp & ~r.x))) | (cq.x & (aq | (hq & ~r.x))),
                      (cp.y & (ap | (hp & ~r.y))) | (cq.y & (aq | (hq & ~r.y))),
                      (cp.z & (ap | (hp & ~r.z))) | (cq.z & (aq | (hq & ~r.z))),
                      (cp.w & (ap | (hp & ~r.w))) | (cq.w & (aq | (hq & ~r.w))));
}

// The decision in any mode.
// slot: sixteen bytes of shared memory per warp where all 32 lanes call together, else nullptr.
// GENERAL: false where DEC_GENERAL is not among the caller's modes.
template <bool WARP = false, bool GENERAL = true>
__device__ __forceinline__ uint4 decide4_mode(int mode, uint4 cp, uint4 cq, Thresh tp, Thresh tq,
                                              Key key, uint32_t qgroup, uint32_t step,
                                              uint32_t stream, uint8_t* slot = nullptr)
{
    if (mode == DEC_NONE || mode == DEC_ONE) return decide4_one(mode, cp, cq, tp, tq, key, qgroup, step, stream);
    if (!GENERAL || mode == DEC_FEW) return decide4_few(cp, cq, tp, tq, key, qgroup, step, stream);
    return decide4<WARP>(cp, cq, tp, tq, key, qgroup, PlaneMaker{step, key}, stream, slot);
}

// Quenched disorder (mcsDisorder2SyncRng): every site carries a 2-bit rate class c (bit 0 in
// d0, bit 1 in d1) that picks thresholds tp[c] / tq[c]; the comparison u < T(site) runs on the
// same random planes as decide4, so equal rates in every class give decide4's result.
struct DisorderRates {
    Thresh tp[4], tq[4];
    int planes;            // most planes any of the eight thresholds can need
    uint32_t last_planes;  // bit k: plane k is the last that one of them, but not the last of all, can need
};

inline DisorderRates make_disorder_rates(const uint64_t Tp[4], const uint64_t Tq[4])
{
    DisorderRates dr{};
    for (int c = 0; c < 4; ++c) {
        dr.tp[c] = make_thresh(Tp[c]);
        dr.tq[c] = make_thresh(Tq[c]);
        if (dr.tp[c].planes > dr.planes) dr.planes = dr.tp[c].planes;
        if (dr.tq[c].planes > dr.planes) dr.planes = dr.tq[c].planes;
        if (dr.tp[c].planes) dr.last_planes |= 1u << (dr.tp[c].planes - 1);
        if (dr.tq[c].planes) dr.last_planes |= 1u << (dr.tq[c].planes - 1);
    }
    if (dr.planes) dr.last_planes &= ~(1u << (dr.planes - 1));  // there, what is left is dropped anyway
    return dr;
}

__device__ __forceinline__ uint32_t sel_class(uint32_t d0, uint32_t d1, uint32_t b0, uint32_t b1, uint32_t b2,
                                              uint32_t b3)
{
    return (~d1 & ((~d0 & b0) | (d0 & b1))) | (d1 & ((~d0 & b2) | (d0 & b3)));
}

__device__ __forceinline__ uint32_t dis_word(uint32_t cp, uint32_t cq, uint32_t d0, uint32_t d1,
                                             const uint32_t bp[4], const uint32_t bq[4])
{
    return (cp & sel_class(d0, d1, bp[0], bp[1], bp[2], bp[3])) |
           (cq & sel_class(d0, d1, bq[0], bq[1], bq[2], bq[3]));
}

template <class Planes>
__device__ __forceinline__ uint4 decide4_dis(uint4 cp, uint4 cq, uint4 d0, uint4 d1, const DisorderRates& dr,
                                             Key key, uint32_t qgroup, const Planes& planes, uint32_t stream,
                                             uint8_t* slot)
{
    uint32_t ap[4], aq[4], hp[4], hq[4];
    for (int c = 0; c < 4; ++c) {
        ap[c] = dr.tp[c].always ? 0xFFFFFFFFu : 0u;
        aq[c] = dr.tq[c].always ? 0xFFFFFFFFu : 0u;
        hp[c] = dr.tp[c].planes ? 0xFFFFFFFFu : 0u;
        hq[c] = dr.tq[c].planes ? 0xFFFFFFFFu : 0u;
    }
    // decided flips (threshold 2^32) and sites still equal to their threshold's prefix
    const uint4 flip = make_uint4(dis_word(cp.x, cq.x, d0.x, d1.x, ap, aq), dis_word(cp.y, cq.y, d0.y, d1.y, ap, aq),
                                  dis_word(cp.z, cq.z, d0.z, d1.z, ap, aq), dis_word(cp.w, cq.w, d0.w, d1.w, ap, aq));
    const uint4 eq = make_uint4(dis_word(cp.x, cq.x, d0.x, d1.x, hp, hq), dis_word(cp.y, cq.y, d0.y, d1.y, hp, hq),
                                dis_word(cp.z, cq.z, d0.z, d1.z, hp, hq), dis_word(cp.w, cq.w, d0.w, d1.w, hp, hq));
    // threshold bit of every site's class and kind of candidate
    auto pick = [&](const uint32_t bp[4], const uint32_t bq[4]) {
        auto one = [&](uint32_t c, uint32_t e0, uint32_t e1) {
            return (c & sel_class(e0, e1, bq[0], bq[1], bq[2], bq[3])) |
                   (~c & sel_class(e0, e1, bp[0], bp[1], bp[2], bp[3]));
        };
        return make_uint4(one(cq.x, d0.x, d1.x), one(cq.y, d0.y, d1.y), one(cq.z, d0.z, d1.z), one(cq.w, d0.w, d1.w));
    };
    auto tb = [&](int k) {
        uint32_t bp[4], bq[4];
        for (int c = 0; c < 4; ++c) {
            bp[c] = (uint32_t)((int32_t)(dr.tp[c].t << k) >> 31);
            bq[c] = (uint32_t)((int32_t)(dr.tq[c].t << k) >> 31);
        }
        return pick(bp, bq);
    };
    auto drop = [&](int k, uint4& e, uint4& f) {
        if (!((dr.last_planes >> k) & 1u)) return;
        uint32_t kp[4], kq[4];
        for (int c = 0; c < 4; ++c) {
            kp[c] = k + 1 == dr.tp[c].planes ? 0u : 0xFFFFFFFFu;
            kq[c] = k + 1 == dr.tq[c].planes ? 0u : 0xFFFFFFFFu;
        }
        const uint4 keep = pick(kp, kq);
        f.x &= ~(e.x & ~keep.x);
        f.y &= ~(e.y & ~keep.y);
        f.z &= ~(e.z & ~keep.z);
        f.w &= ~(e.w & ~keep.w);
        e.x &= keep.x;
        e.y &= keep.y;
        e.z &= keep.z;
        e.w &= keep.w;
    };
    return decide_planes<true>(eq, flip, dr.planes, key, group_part(qgroup, stream, key), planes, tb, drop, slot);
}

__device__ __forceinline__ uint4 operator^(uint4 a, uint4 b)
{
    return make_uint4(a.x ^ b.x, a.y ^ b.y, a.z ^ b.z, a.w ^ b.w);
}

}  // namespace kpzb
