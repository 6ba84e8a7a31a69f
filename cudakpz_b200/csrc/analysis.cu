// analysis.cu -- height reconstruction, roughness moments, correlator and lattice
// invariants on ENC_CBBIT lattices (sm_100a).
//
// Heights follow the reference's path walk (kpz/correlator.cpp:47-96, :337-399):
//   row y starts at Hs(y) = h(0,y-1) + (2*s_y(0,y)-1) with h(0,-1) = 0, walks x = 1..L-1
//   adding 2*s_x(x,y)-1, and the wrap adds 2*s_x(0,y)-1 giving h(0,y) = Hs(y) + rowsum(y).
// Moments: S1 and S2 exact in int64, S3..S7 in FP64 from exact integer counts (below); ch uses
// the exact int64 cross sum; cs counts equal minus different slope bits
// (kpz/correlator.cpp:463-477).
// Invariants extend SchedulerService::consitencyCheck (kpz/schedulerService.cpp:733-854)
// to ENC_CBBIT: x-slope row sums, y-slope column sums, plaquette loops.
//
// Two launches: (1) row_kernel: per-row slope counts and the row starts within a block of rows;
// (2) walk_kernel: the walk in groups of eight sites from the block totals on, whose last CTA adds
// the per-CTA partials in a fixed order, so the FP64 sums are deterministic.
#include <cstring>
#include <map>
#include <mutex>
#include "kpzb_api_internal.h"
#include "kpzb_common.cuh"
#include "kpzb_internal.h"

namespace kpzb {

constexpr int AN_MAX_GRID = 148;  // CTAs of the walk: one per SM of a B200
constexpr int AN_ROW_THREADS = 256;
// Lattices of at least 128 words per quadrant row are walked in four parts per row, each by its
// own warp: 16384^2 is then 13.8 parts per warp instead of 3.5 rows (a last wave 1.3 % short
// instead of 14 %).
constexpr int AN_PART_WORDS = 128;

struct Partial {
    long long s1, s2, hmin, hmax, cross, agree, snap_s1, pad;
    double s[5];
    double pad2[3];
};

// Per-row record w: x-slope row sum (even) with the y-slope bit of x = 0 in bit 0.  Rows of at least
// AN_PART_WORDS words have {n1, n2, n3, w} with the X-slope bits set in the row's first one, two and
// three quarters; the others only w, since tall lattices have many of them (4 bytes a row instead of
// 16 are 24 GiB of a lattice of 2^8 x 2^30).
__host__ __device__ constexpr bool long_rows(int lx) { return (1ull << lx) >= 64ull * AN_PART_WORDS; }
__host__ __device__ constexpr int row_ints(int lx) { return long_rows(lx) ? 4 : 1; }
__device__ __forceinline__ int row_word(const int* rowinfo, uint64_t y, int lx)
{
    return rowinfo[(y + 1) * row_ints(lx) - 1];
}
__device__ __forceinline__ int row_sum(int w) { return w & ~1; }
__device__ __forceinline__ int row_ystep(int w) { return 2 * (w & 1) - 1; }

// Rows are scanned in up to AN_MAX_BLOCKS blocks of 2^lgb rows: rowstart[y] is relative to the
// start of y's block, and the block's record holds its total step and the extremes of its starts.
constexpr int AN_MAX_BLOCKS = 256;
struct RowBlock {
    long long total, lo, hi;
};
__host__ __device__ constexpr int row_block_lg(int ly) { return ly <= 12 ? (ly < 4 ? ly : 4) : ly - 8; }

// What the kernels leave in the scratch beside the partial sums: the row blocks of the system and
// of the snapshot, and the walk's last-CTA ticket (cleared by every row_kernel, so a count left
// over by callers that raced on a shared scratch does not outlive the next call).
struct WalkState {
    RowBlock block[2][AN_MAX_BLOCKS];
    unsigned int ticket;
};

// Exclusive scan of one int64 per thread over a CTA of NT threads; *total = the sum.
template <int NT>
__device__ __forceinline__ long long cta_exclusive_scan(long long v, long long* total)
{
    __shared__ long long wsum[NT / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    long long incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long a = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += a;
    }
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    long long before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) {
        const long long s = wsum[w];
        if (w < wid) before += s;
        all += s;
    }
    __syncthreads();
    *total = all;
    return before + incl - v;
}

__host__ inline bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

// Four words from p on: one 128-bit load, or word by word.
template <bool WORDS>
__device__ __forceinline__ uint4 load_words4(const uint32_t* p)
{
    if (WORDS) return make_uint4(p[0], p[1], p[2], p[3]);
    return *reinterpret_cast<const uint4*>(p);
}

// ---- launch 1: per-row slope counts and row starts within a block of rows ----
// A CTA takes one block of rows; blockIdx.y picks the lattice (the system, the snapshot).  A warp
// reads a row's 2 Wr words as 128-bit loads, ordered quarter by quarter and both X quadrants of
// a quarter together, so that every lane has a load of every step; rows shorter than
// AN_PART_WORDS take Wr / 2 lanes each.  A caller's own lattice may start at any word
// (kpzb_roughness_noalloc, kpzb_gram_add_device): off a 16-byte boundary the instance WORDS reads
// the same 16 bytes word by word.  The scan over blocks is left to each reader, which needs
// no grid-wide step: a scan of all rows by one CTA (a launch of its own, or the last CTA here)
// took 15 to 27 us at 8192 and 16384 rows, most of both kernels' time.
template <bool WORDS>
__global__ void __launch_bounds__(AN_ROW_THREADS)
row_kernel(const uint32_t* __restrict__ sys0, const uint32_t* __restrict__ sys1, int lx, int ly,
           int* __restrict__ rowinfo0, int64_t* __restrict__ rowstart0, WalkState* ws)
{
    __shared__ int w_s[AN_ROW_THREADS];
    __shared__ long long lo_s[AN_ROW_THREADS / 32], hi_s[AN_ROW_THREADS / 32];
    const uint64_t Wr = 1ull << (lx - 6);
    const uint64_t Q = 1ull << (lx + ly - 6);
    const uint64_t rows = 1ull << ly;
    const uint32_t* sys = blockIdx.y ? sys1 : sys0;
    int* rowinfo = rowinfo0 + blockIdx.y * rows * row_ints(lx);
    int64_t* rowstart = rowstart0 + blockIdx.y * rows;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    constexpr int NWARP = AN_ROW_THREADS / 32;
    const int lgb = row_block_lg(ly);
    const uint64_t yb = (uint64_t)blockIdx.x << lgb, ye = yb + (1ull << lgb);
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) ws->ticket = 0u;
    auto count4 = [](uint4 v) { return __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w); };
    auto load4 = [](const uint32_t* r, uint64_t i) { return load_words4<WORDS>(r + 4 * i); };
    // site (0,y) lies on sublattice y&1, word 0, bit 0
    auto sy0 = [&](uint64_t y) { return (int)(sys[((y & 1) ? 2 * Q : 0) + Q + y * Wr] & 1u); };
    long long carry = 0, lo = 0x7fffffffffffffffll, hi = -0x7fffffffffffffffll;
    for (uint64_t base = yb; base < ye; base += AN_ROW_THREADS) {
        const uint64_t end = ye - base < AN_ROW_THREADS ? ye : base + AN_ROW_THREADS;
        auto put = [&](uint64_t y, int n1, int n2, int n3, int n, int s) {
            const int w = (int)(2 * (int64_t)n - (int64_t)(1ull << lx)) | s;
            if (long_rows(lx)) reinterpret_cast<int4*>(rowinfo)[y] = make_int4(n1, n2, n3, w);
            else rowinfo[y] = w;
            w_s[y - base] = w;
        };
        if (Wr >= AN_PART_WORDS) {
            const uint64_t qv = Wr / 16;  // 128-bit loads per quadrant row quarter (at least 8)
#pragma unroll 2
            for (uint64_t y = base + wid; y < end; y += NWARP) {
                const int s = sy0(y);
                const uint32_t* r0 = sys + y * Wr;
                const uint32_t* r1 = sys + 2 * Q + y * Wr;
                int n[4] = {0, 0, 0, 0};
                if (qv == 8) {  // a step of the warp covers two quarters
                    uint4 v[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) v[h] = load4(lane & 8 ? r1 : r0, 16 * h + 8 * (lane >> 4) + (lane & 7));
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int c = count4(v[h]);
                        n[2 * h] = lane < 16 ? c : 0;
                        n[2 * h + 1] = lane < 16 ? 0 : c;
                    }
                } else {
                    for (uint64_t i = lane; i < 2 * qv; i += 32) {
                        uint4 v[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) v[q] = i >= qv ? load4(r1, q * qv + i - qv) : load4(r0, q * qv + i);
#pragma unroll
                        for (int q = 0; q < 4; ++q) n[q] += count4(v[q]);
                    }
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) n[q] = __reduce_add_sync(0xffffffffu, n[q]);
                if (lane == 0) put(y, n[0], n[0] + n[1], n[0] + n[1] + n[2], n[0] + n[1] + n[2] + n[3], s);
            }
        } else {
            const int sw = (int)(Wr / 2), rpw = 32 / sw;  // lanes per row, rows per warp (powers of two)
            for (uint64_t y0 = base + (uint64_t)wid * rpw; y0 < end; y0 += (uint64_t)NWARP * rpw) {
                const uint64_t y = y0 + lane / sw;
                const int j = lane % sw, half = sw / 2;
                const bool in = y < end;
                const int s = in ? sy0(y) : 0;
                int n = in ? count4(load4(sys + (j >= half ? 2 * Q : 0) + y * Wr, j % half)) : 0;
                for (int o = 1; o < sw; o <<= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
                if (in && j == 0) put(y, 0, 0, 0, n, s);
            }
        }
        if (!rowstart0) continue;  // counts only
        __syncthreads();
        // Hs(y) = sum_{y'<=y} ystep(y') + sum_{y'<y} rowsum(y')
        const uint64_t y = base + threadIdx.x;
        const int w = y < end ? w_s[threadIdx.x] : 0;
        const long long v = y < end ? row_ystep(w) + row_sum(w) : 0;
        long long total;
        const long long start = carry + cta_exclusive_scan<AN_ROW_THREADS>(v, &total) + row_ystep(w);
        if (y < end) {
            rowstart[y] = start;
            lo = min(lo, start);
            hi = max(hi, start);
        }
        carry += total;
    }
    if (!rowstart0) return;
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) {
        lo_s[wid] = lo;
        hi_s[wid] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < NWARP; ++w) {
            lo = min(lo, lo_s[w]);
            hi = max(hi, hi_s[w]);
        }
        ws->block[blockIdx.y][blockIdx.x] = RowBlock{carry, lo, hi};
    }
}

// Heights at the start of every row block into base_s (an array of AN_MAX_BLOCKS in shared
// memory) and the middle of the row starts; NT >= AN_MAX_BLOCKS threads, all of them.
template <int NT>
__device__ __forceinline__ long long row_block_bases(const RowBlock* blocks, int nblk, long long* base_s)
{
    __shared__ long long lo_s[NT / 32], hi_s[NT / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    RowBlock b{0, 0x7fffffffffffffffll, -0x7fffffffffffffffll};
    const bool in = (int)threadIdx.x < nblk;
    if (in) b = blocks[threadIdx.x];
    long long total;
    const long long base = cta_exclusive_scan<NT>(b.total, &total);
    if (in) {
        base_s[threadIdx.x] = base;
        b.lo += base;
        b.hi += base;
    }
    if (wid < AN_MAX_BLOCKS / 32)
        for (int o = 16; o > 0; o >>= 1) {
            b.lo = min(b.lo, __shfl_xor_sync(0xffffffffu, b.lo, o));
            b.hi = max(b.hi, __shfl_xor_sync(0xffffffffu, b.hi, o));
        }
    if (lane == 0) {
        lo_s[wid] = b.lo;
        hi_s[wid] = b.hi;
    }
    __syncthreads();
    long long lo = lo_s[0], hi = hi_s[0];
#pragma unroll
    for (int w = 1; w < AN_MAX_BLOCKS / 32; ++w) {
        lo = min(lo, lo_s[w]);
        hi = max(hi, hi_s[w]);
    }
    __syncthreads();
    return (lo + hi) >> 1;
}

// ---- launch 2: the walk ----
//
// A group of eight sites is its height H before the first site and an 8-bit slope pattern, so
// the sums of h^k over the lattice follow from counts of (H, pattern) alone.  Each CTA keeps the
// counts of WALK_BINS heights of one parity x 256 patterns in shared memory and adds one per
// group: 27 instructions for eight sites, one of them a shared atomic, where evaluating the powers
// site by site took about 17 a site (330 us against 49 us at 2^28 sites, 70 against 25 at 2^26).  The
// integer ALU bounds it (76 % active at 2^30 sites; the atomics, 4.8 wavefronts each, keep shared
// memory half busy).  The even rows' groups all have heights of one parity and the odd rows' of the
// other, so a CTA walks rows of one parity and a bin covers two heights.  At the end thread (pattern
// p, slice of heights) takes the power sums of H over its bins and combines them with the pattern's
// own offsets' power sums.
//
// Counts are exact and the bins' heights span less than 2^9, so every term up to k = 7 of a
// surface with |H| <= 16 is an exact integer in FP64; above that the terms of one bin do not
// cancel (offsets within a group are at most 8).
//
// The bins cover WALK_REACH heights on each side of the middle of the row starts (a surface of
// 16384^2 has heights within about 30 of its mean at t = 10^4).  A chunk of 64 sites that leaves
// them goes by its own power sums (walk_far), as does a row's first chunk when the row's slopes
// do not close.
constexpr int WALK_BINS = 192;
constexpr int WALK_REACH = WALK_BINS - 64;  // a chunk moves at most 64 from its first height
constexpr int WALK_LUT = 256;
constexpr int WALK_SMEM = WALK_BINS * 256 * 4;

// Number of set bits of each byte.
__device__ __forceinline__ uint32_t byte_popc(uint32_t v)
{
    v -= (v >> 1) & 0x55555555u;
    v = (v & 0x33333333u) + ((v >> 2) & 0x33333333u);
    return (v + (v >> 4)) & 0x0F0F0F0Fu;
}

// One word of a Partial: its value over the CTA's threads, by the warp that reads it.  Words 0, 1
// and 4-6 are added as integers, 2 and 3 are the extremes, the rest are added in FP64.
constexpr int PARTIAL_SUMS = 12;
__device__ __forceinline__ int partial_word(int q) { return q < 7 ? q : q + 1; }

// Reduce a Partial per thread to *out: every thread stores its twelve values to buf (in shared
// memory, 12 * NT words) and a warp adds up each quantity, lane by lane and then by a tree, in the
// same order in every call.  (Shuffling all twelve 64-bit values through every warp took 4 us.)
template <int NT>
__device__ __forceinline__ void put_partial(const Partial& p, long long* buf)
{
    const long long* pw = reinterpret_cast<const long long*>(&p);
#pragma unroll
    for (int q = 0; q < PARTIAL_SUMS; ++q) buf[q * NT + threadIdx.x] = pw[partial_word(q)];
}

// The same values added to what this thread has stored.
template <int NT>
__device__ __forceinline__ void add_partial(const Partial& p, long long* buf)
{
    const long long* pw = reinterpret_cast<const long long*>(&p);
#pragma unroll
    for (int q = 0; q < PARTIAL_SUMS; ++q) {
        long long& v = buf[q * NT + threadIdx.x];
        const long long x = pw[partial_word(q)];
        v = q == 2 ? min(v, x) : q == 3 ? max(v, x) : q < 7 ? v + x : __double_as_longlong(__longlong_as_double(v) + __longlong_as_double(x));
    }
}

template <int NT>
__device__ __forceinline__ void cta_reduce(const long long* buf, Partial* out)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (wid < PARTIAL_SUMS) {
        const long long* v = buf + wid * NT + lane;
        long long* o = reinterpret_cast<long long*>(out) + partial_word(wid);
        if (wid >= 7) {
            double s = 0.0;
            for (int i = 0; i < NT; i += 32) s += __longlong_as_double(v[i]);
            for (int k = 16; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
            if (lane == 0) *o = __double_as_longlong(s);
        } else {
            const bool lo = wid == 2, hi = wid == 3;
            long long s = v[0];
            auto merge = [&](long long x) { s = lo ? min(s, x) : hi ? max(s, x) : s + x; };
            for (int i = 32; i < NT; i += 32) merge(v[i]);
            for (int k = 16; k > 0; k >>= 1) merge(__shfl_xor_sync(0xffffffffu, s, k));
            if (lane == 0) *o = s;
        }
    }
    __syncthreads();
}

__device__ __forceinline__ Partial empty_partial()
{
    Partial p{};
    p.hmin = 0x7fffffffffffffffll;
    p.hmax = -0x7fffffffffffffffll;
    return p;
}

// What a warp of the walk needs to find the chunks of its items: rows of parity `par`, or quarters of
// them where rows are long.
struct WalkGeom {
    const uint32_t *sys, *snap;
    const int* rowinfo;       // records of the system's rows, then of the snapshot's
    const int64_t* rowstart;
    const long long *base, *base_s;  // heights at the start of every row block
    const uint32_t* step4;           // table of add_chunk
    long long mid, mid_s;            // middles of the row starts
    int lx, ly, par;
    uint64_t item, step;  // the warp's first item and the distance to its next
};

// Items of one row parity.
__host__ __device__ inline uint64_t walk_items(int lx, int ly)
{
    const uint64_t Wr = 1ull << (lx - 6), rows = 1ull << ly;
    return Wr >= AN_PART_WORDS ? 2 * rows : rows / 2 / (Wr < 32 ? 32 / Wr : 1);
}

// One chunk of 64 sites: its X-slope words (even-x and odd-x), the height before it relative to
// the middle of the row starts, and the same of the snapshot; first: it starts at x = 0.
struct Chunk {
    uint32_t e, o, es, os;
    long long rel, rel_s;
    int sum_r, sum_s;  // slope sums of the chunk's row
    bool first;
    __device__ bool binned() const { return rel >= -WALK_REACH && rel < WALK_REACH && !(first && sum_r != 0); }
    // u and v as bytes: no carry while the chunk stays within [-127, 127] of the middles
    __device__ bool bytes() const
    {
        return rel >= -63 && rel <= 63 && rel_s >= -63 && rel_s <= 63 && !(first && (sum_r | sum_s) != 0);
    }
};

// Hands every chunk of the warp's items to `chunk`, with the number of agreeing Y slopes.
template <bool CORR, class F>
__device__ __forceinline__ void walk_chunks(const WalkGeom& g, F&& chunk)
{
    const uint64_t Wr = 1ull << (g.lx - 6);
    const uint64_t Q = 1ull << (g.lx + g.ly - 6);
    const uint64_t rows = 1ull << g.ly;
    const int lane = threadIdx.x & 31, lgb = row_block_lg(g.ly);
    const int wl = (int)(Wr < 32 ? Wr : 32);      // lanes per row
    const int rpw = 32 / wl;                      // rows per warp
    const int parts = Wr >= AN_PART_WORDS ? 4 : 1;
    const uint64_t pw = Wr / parts;               // words per part
    const uint64_t items = walk_items(g.lx, g.ly);
    const int sub = lane % wl;
    const uint64_t be = g.par ? 2 * Q : 0, bo = g.par ? 0 : 2 * Q;

    for (uint64_t it = g.item; it < items; it += g.step) {
        const int part = (int)(it % parts);
        const uint64_t y = 2 * (it / parts * rpw + lane / wl) + g.par;
        const uint64_t off = y * Wr + part * pw;
        const uint32_t *pe = g.sys + be + off, *po = g.sys + bo + off;
        const uint32_t *qe = g.snap + be + off, *qo = g.snap + bo + off;
        // the next chunk's words: X of both sublattices, for the correlator Y and the snapshot's
        uint32_t w[CORR ? 8 : 2];
        auto load = [&](uint64_t c) {
            w[0] = pe[c];
            w[1] = po[c];
            if (CORR) {
                w[2] = qe[c];
                w[3] = qo[c];
                w[4] = pe[Q + c];
                w[5] = po[Q + c];
                w[6] = qe[Q + c];
                w[7] = qo[Q + c];
            }
        };
        load(sub);
        // height before the part's first site: Hs - e0 + 2 (bits set before it) - sites
        auto record = [&](uint64_t i) {
            return parts > 1 ? reinterpret_cast<const int4*>(g.rowinfo)[i] : make_int4(0, 0, 0, g.rowinfo[i]);
        };
        auto before = [&](const int4& r) { return part == 0 ? 0 : part == 1 ? r.x : part == 2 ? r.y : r.z; };
        const long long back = (long long)(64 * pw * part);
        const int4 ri = record(y);
        long long H = g.rowstart[y] + g.base[y >> lgb] - (2 * (int)(g.sys[be + y * Wr] & 1u) - 1) +
                      2 * (long long)before(ri) - back - g.mid;
        long long Hsn = 0;
        Chunk ch{};
        ch.sum_r = row_sum(ri.w);
        if (CORR) {
            const int4 si = record(rows + y);
            ch.sum_s = row_sum(si.w);
            Hsn = g.rowstart[rows + y] + g.base_s[y >> lgb] - (2 * (int)(g.snap[be + y * Wr] & 1u) - 1) +
                  2 * (long long)before(si) - back - g.mid_s;
        }
        for (uint64_t c = sub; c < pw; c += wl) {
            ch.e = w[0];
            ch.o = w[1];
            int eq = 0;
            if (CORR) {
                ch.es = w[2];
                ch.os = w[3];
                eq = __popc(~(w[4] ^ w[6])) + __popc(~(w[5] ^ w[7]));
            }
            if (c + wl < pw) load(c + wl);
            // the chunk's total step and the heights before it, in the row's lanes
            const int n = __popc(ch.e) + __popc(ch.o) - 32;
            int incl = n;
            int ns = 0, incl_s = 0;
            if (CORR) incl_s = ns = __popc(ch.es) + __popc(ch.os) - 32;
            for (int k = 1; k < wl; k <<= 1) {
                const int a = __shfl_up_sync(0xffffffffu, incl, k, wl);
                if (sub >= k) incl += a;
                if (CORR) {
                    const int b = __shfl_up_sync(0xffffffffu, incl_s, k, wl);
                    if (sub >= k) incl_s += b;
                }
            }
            ch.first = part == 0 && c == 0;
            ch.rel = H + 2 * (incl - n);
            H += 2 * __shfl_sync(0xffffffffu, incl, wl - 1, wl);
            if (CORR) {
                ch.rel_s = Hsn + 2 * (incl_s - ns);
                Hsn += 2 * __shfl_sync(0xffffffffu, incl_s, wl - 1, wl);
            }
            chunk(ch, eq);
        }
    }
}

// A chunk of 64 sites outside the bins: its heights are b + d_i with b the height before its first
// site and |d_i| <= 64, so the power sums of d are whole numbers below 2^49, exact in FP64, and the
// sums of h^k follow once per chunk by the binomial expansion.  The d_i come four at a time as biased
// bytes from a table of the four-site patterns (even-x bits in bits 0-1, odd-x bits in bits 2-3).
// Nine FP64 and about six integer operations a site on two pipes, where powers in 32- and 64-bit
// integers kept one pipe busy for about 40 cycles a warp.  open: the chunk's first site is x = 0 of a
// row whose slopes sum to `row`, not 0; its height is b + d_0 + row, the one its row ends with, and it
// is left out of the power sums.
__device__ __forceinline__ void add_chunk(Partial& s, uint32_t e, uint32_t o, long long b, bool open, int row,
                                          const uint32_t* step4)
{
    const uint32_t A = (e & 0x33333333u) | ((o & 0x33333333u) << 2), B = ((e >> 2) & 0x33333333u) | (o & 0xCCCCCCCCu);
    int a1 = 0, a2 = 0, dmin = 255, dmax = 0;
    double A3 = 0, A4 = 0, A5 = 0, A6 = 0, A7 = 0;
    uint32_t base = 0x7C7C7C7Cu;  // bytes: d before the four sites, + 128 - 4 (the table's bias)
#pragma unroll 4
    for (int g = 0; g < 16; ++g) {
        const uint32_t u = base + step4[((g & 1 ? B : A) >> (4 * (g >> 1))) & 15u];
        base = __byte_perm(u, 0u, 0x3333) - 0x04040404u;
        const int x = (int)(u ^ 0x80808080u);  // the four d as signed bytes
        a1 = __dp4a(x, 0x01010101, a1);
        a2 = __dp4a(x, x, a2);
        int v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            v[j] = (int)__byte_perm(u, 0u, 0x4440 | j);  // d + 128
            const double d = __hiloint2double(0x43300000, v[j]) - 4503599627370624.0;  // 2^52 + 128
            const double d2 = d * d, d4 = d2 * d2, d5 = d4 * d;
            A3 += d2 * d;
            A4 += d4;
            A5 += d5;
            A6 += d4 * d2;
            A7 += d5 * d2;
        }
        const int v0 = g == 0 && open ? v[1] : v[0];
        dmin = __vimin3_s32(__vimin3_s32(dmin, v0, v[1]), v[2], v[3]);
        dmax = __vimax3_s32(__vimax3_s32(dmax, v0, v[1]), v[2], v[3]);
    }
    dmin -= 128;
    dmax -= 128;
    const int first = 2 * (int)(e & 1u) - 1;  // d_0
    if (open) {
        a1 -= first;
        a2 -= 1;
        A3 -= first;
        A4 -= 1;
        A5 -= first;
        A6 -= 1;
        A7 -= first;
    }
    const int n = open ? 63 : 64;
    s.s1 += (long long)n * b + a1;
    s.s2 += (long long)n * b * b + 2 * b * a1 + a2;
    s.hmin = min(s.hmin, b + dmin);
    s.hmax = max(s.hmax, b + dmax);
    const double B1 = (double)b, B2 = B1 * B1, B3 = B2 * B1, B4 = B2 * B2, B5 = B4 * B1, B6 = B3 * B3, B7 = B6 * B1;
    const double N = n, A1 = a1, A2 = a2;
    s.s[0] += N * B3 + 3.0 * B2 * A1 + 3.0 * B1 * A2 + A3;
    s.s[1] += N * B4 + 4.0 * B3 * A1 + 6.0 * B2 * A2 + 4.0 * B1 * A3 + A4;
    s.s[2] += N * B5 + 5.0 * B4 * A1 + 10.0 * B3 * A2 + 10.0 * B2 * A3 + 5.0 * B1 * A4 + A5;
    s.s[3] += N * B6 + 6.0 * B5 * A1 + 15.0 * B4 * A2 + 20.0 * B3 * A3 + 15.0 * B2 * A4 + 6.0 * B1 * A5 + A6;
    s.s[4] += N * B7 + 7.0 * B6 * A1 + 21.0 * B5 * A2 + 35.0 * B4 * A3 + 35.0 * B3 * A4 + 21.0 * B2 * A5 + 7.0 * B1 * A6 + A7;
    if (open) {
        const long long hf = b + first + row;
        const double h = (double)hf, h2 = h * h, h3 = h2 * h;
        s.s1 += hf;
        s.s2 += hf * hf;
        s.s[0] += h3;
        s.s[1] += h2 * h2;
        s.s[2] += h3 * h2;
        s.s[3] += h3 * h3;
        s.s[4] += h3 * h3 * h;
        s.hmin = min(s.hmin, hf);
        s.hmax = max(s.hmax, hf);
    }
}

// Sums over a chunk of u v (x) and of v (y), u = 128 + rel + d_i and v = 128 + rel_s + d'_i from the steps
// of the two lattices' slope words; x = 0 takes the height its row ends with, the row's sum further.
__device__ __forceinline__ void add_cross(longlong2& sum, const Chunk& c)
{
    int d = 0, ds = 0, sd = 0, sds = 0, sdd = 0;
    auto add = [&](uint32_t b, uint32_t bs) {
        d += 2 * (int)(b & 1u) - 1;
        ds += 2 * (int)(bs & 1u) - 1;
        sd += d;
        sds += ds;
        sdd += d * ds;
    };
#pragma unroll 4
    for (int i = 0; i < 32; ++i) {
        add(c.e >> i, c.es >> i);
        add(c.o >> i, c.os >> i);
    }
    const long long r = 128 + c.rel, q = 128 + c.rel_s;
    sum.x += 64 * r * q + r * sds + q * sd + sdd;
    sum.y += 64 * q + sds;
    if (c.first) {
        const long long u = r + 2 * (int)(c.e & 1u) - 1, v = q + 2 * (int)(c.es & 1u) - 1;
        sum.x += (u + c.sum_r) * (v + c.sum_s) - u * v;
        sum.y += c.sum_s;
    }
}

// The chunks that the walk over the bins leaves out, in a second walk by the warps that met one: as
// code of that walk they cost a tenth of its time in registers, although surfaces in their growth
// regime have none.  A pyramid of 16384^2, nearly all of it outside the bins: roughness 310 us, a
// correlation of random words 470 us (490 and 950 with the powers of every height in the first walk;
// 330 and 690 by chunks alone, without bins).  cross: the correlator's sums of u v and v over the
// chunks without bytes.
template <bool CORR>
__device__ __noinline__ void walk_far(const WalkGeom& g, Partial* sums, longlong2* cross)
{
    walk_chunks<CORR>(g, [&](const Chunk& c, int) {
        if (!c.binned()) add_chunk(*sums, c.e, c.o, c.rel + g.mid, c.first && c.sum_r != 0, c.sum_r, g.step4);
        if (CORR && !c.bytes()) add_cross(*cross, c);
    });
}

// CORR: also the correlator's sums against `snap` (cross sum of heights, agreeing slopes).  Its
// heights relative to the two lattices' middles are built as biased bytes from a table of
// the patterns' cumulative steps and multiplied four sites at a time (dp4a).
constexpr int walk_threads(bool corr) { return corr ? 768 : 1024; }  // 85 and 64 registers

template <bool CORR>
__global__ void __launch_bounds__(walk_threads(CORR), 1)
walk_kernel(const uint32_t* __restrict__ sys, const uint32_t* __restrict__ snap, int lx, int ly,
            const int* __restrict__ rowinfo, const int64_t* __restrict__ rowstart, Partial* __restrict__ partials,
            Partial* __restrict__ out, WalkState* ws)
{
    constexpr int NT = walk_threads(CORR), NWARP = NT / 32;
    extern __shared__ __align__(16) uint32_t hist[];  // [height bin][pattern ^ bin]
    __shared__ uint2 lut[CORR ? WALK_LUT : 1];
    __shared__ long long base_s[CORR ? 2 : 1][AN_MAX_BLOCKS];
    __shared__ uint32_t step4[16];
    __shared__ int used[2];  // first and last bin of a chunk's first group
    __shared__ bool last;

    const uint64_t rows = 1ull << ly;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int par = (int)(blockIdx.x & 1);            // row parity of this CTA
    const uint64_t nctas = gridDim.x >> 1, cta = blockIdx.x >> 1;

    if (threadIdx.x == 0) {
        used[0] = WALK_BINS;
        used[1] = -1;
    }
    for (int i = threadIdx.x; i < WALK_BINS * 64; i += NT) reinterpret_cast<uint4*>(hist)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (CORR && threadIdx.x < WALK_LUT) {
        // byte j: 8 + sum_{k <= j} (2 bit_k - 1), the pattern's even-x bits low, odd-x bits high
        int cum = 8;
        uint32_t w[2] = {0u, 0u};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            cum += 2 * (int)((threadIdx.x >> ((j & 1 ? 4 : 0) + (j >> 1))) & 1u) - 1;
            w[j >> 2] |= (uint32_t)cum << (8 * (j & 3));
        }
        lut[threadIdx.x] = make_uint2(w[0], w[1]);
    }
    if (threadIdx.x < 16) {
        // byte j: 4 + sum_{k <= j} (2 bit_k - 1)
        int cum = 4;
        uint32_t w = 0;
        for (int j = 0; j < 4; ++j) {
            cum += 2 * (int)((threadIdx.x >> ((j & 1 ? 2 : 0) + (j >> 1))) & 1u) - 1;
            w |= (uint32_t)cum << (8 * j);
        }
        step4[threadIdx.x] = w;
    }
    const int lgb = row_block_lg(ly), nblk = (int)(rows >> lgb);
    const long long mid = row_block_bases<NT>(ws->block[0], nblk, base_s[0]);
    const long long mid_s = CORR ? row_block_bases<NT>(ws->block[1], nblk, base_s[CORR ? 1 : 0]) : 0;
    // bin s holds groups with height H0 + 2 s before their first site; H0 has the parity of the
    // heights before x = 0 of this CTA's rows, Hs(y) - e0
    const long long first_h = rowstart[par] - 1;  // block 0 starts at 0; e0 = +-1: either way the same parity
    const long long H0 = mid - WALK_BINS + ((mid - WALK_BINS - first_h) & 1);
    const int h0_rel = (int)(mid - H0);
    __syncthreads();

    int bin_lo = WALK_BINS, bin_hi = -1;
    bool far = false;  // this lane has met a chunk that the bins (or the correlator's bytes) do not reach
    // correlator: sums over sites of u v and of v, u = h - mid + 128 and v = h' - mid' + 128
    long long uv_sum = 0, v_sum = 0, agree = 0;

    // items are dealt to the CTAs in turn, so that few of them still use every SM (2^20 x 2^8 sites:
    // roughness 210 -> 135 us)
    const WalkGeom geom{sys, snap, rowinfo, rowstart, base_s[0], base_s[CORR ? 1 : 0], step4, mid, mid_s, lx, ly, par,
                        (uint64_t)wid * nctas + cta, nctas * NWARP};
    walk_chunks<CORR>(geom, [&](const Chunk& c, int eq) {
        // patterns of the even and the odd groups, a byte each, and their set bits
        const uint32_t A = (c.e & 0x0F0F0F0Fu) | ((c.o & 0x0F0F0F0Fu) << 4);
        const uint32_t B = ((c.e >> 4) & 0x0F0F0F0Fu) | (c.o & 0xF0F0F0F0u);
        const uint32_t pa = byte_popc(A), pb = byte_popc(B);
        if (c.binned()) {
            // absolute bin of each group: s0 + bits before it - 4 per group before it
            const int s0 = ((int)c.rel + h0_rel) >> 1;
            bin_lo = min(bin_lo, s0);
            bin_hi = max(bin_hi, s0);
            const uint32_t sa = (pa + pb) * 0x01010100u + (uint32_t)s0 * 0x01010101u - 0x18100800u;
            const uint32_t sb = sa + pa - 0x04040404u;
            // the pattern is XORed with the bin so that equal patterns at different heights
            // lie in different banks
            const uint32_t xa = A ^ sa, xb = B ^ sb;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t ta = __byte_perm(xa, sa, i ? 0x7362 : 0x5140);
                const uint32_t tb = __byte_perm(xb, sb, i ? 0x7362 : 0x5140);
                atomicAdd(&hist[ta & 0xFFFFu], 1u);
                atomicAdd(&hist[tb & 0xFFFFu], 1u);
                atomicAdd(&hist[ta >> 16], 1u);
                atomicAdd(&hist[tb >> 16], 1u);
            }
        } else {
            far = true;
        }
        if (CORR) {
            agree += 2 * (eq + __popc(~(c.e ^ c.es)) + __popc(~(c.o ^ c.os))) - 128;
            if (c.bytes()) {
                const uint32_t As = (c.es & 0x0F0F0F0Fu) | ((c.os & 0x0F0F0F0Fu) << 4);
                const uint32_t Bs = ((c.es >> 4) & 0x0F0F0F0Fu) | (c.os & 0xF0F0F0F0u);
                uint32_t b = (uint32_t)((int)c.rel + 120) * 0x01010101u, bs = (uint32_t)((int)c.rel_s + 120) * 0x01010101u;
                unsigned int uv = 0, vv = 0;
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                    const uint2 T = lut[((g & 1 ? B : A) >> (8 * (g >> 1))) & 0xFFu];
                    const uint2 Ts = lut[((g & 1 ? Bs : As) >> (8 * (g >> 1))) & 0xFFu];
                    const uint32_t u0 = b + T.x, u1 = b + T.y, v0 = bs + Ts.x, v1 = bs + Ts.y;
                    uv = __dp4a(u0, v0, uv);
                    uv = __dp4a(u1, v1, uv);
                    vv = __dp4a(v0, 0x01010101u, vv);
                    vv = __dp4a(v1, 0x01010101u, vv);
                    // the next group starts at this one's last height: byte 3, less the 8 of the bias
                    b = __byte_perm(u1, 0u, 0x3333) - 0x08080808u;
                    bs = __byte_perm(v1, 0u, 0x3333) - 0x08080808u;
                }
                uv_sum += uv;
                v_sum += vv;
            } else {
                far = true;
            }
        }
    });
    bin_lo = __reduce_min_sync(0xffffffffu, bin_lo);
    bin_hi = __reduce_max_sync(0xffffffffu, bin_hi);
    if (lane == 0) {
        atomicMin(&used[0], bin_lo);
        atomicMax(&used[1], bin_hi);
    }
    __syncthreads();
    Partial acc = empty_partial();
    // thread: pattern p, every (NT / 256)th height bin of those in use (a chunk's later groups
    // start at most 28 bins from its first)
    {
        const int p = (int)(threadIdx.x & 255u);
        const int end = min(used[1] + 29, WALK_BINS);
        unsigned long long n0 = 0, n1 = 0, n2 = 0;  // sums of n, n s, n s^2
        double m3 = 0, m4 = 0, m5 = 0, m6 = 0, m7 = 0;
        int smin = WALK_BINS, smax = -1;
        for (int s = max(used[0] - 28, 0) + (int)(threadIdx.x >> 8); s < end; s += NT / 256) {
            const uint32_t n = hist[s * 256 + (p ^ s)];
            if (n == 0u) continue;
            smin = min(smin, s);
            smax = s;
            n0 += n;
            n1 += (unsigned long long)n * (uint32_t)s;
            n2 += (unsigned long long)n * (uint32_t)(s * s);
            const double d = (double)(H0 + 2 * s), d2 = d * d, N = (double)n * (d2 * d);
            m3 += N;
            m4 += N * d;
            m5 += N * d2;
            m6 += N * (d2 * d);
            m7 += N * (d2 * d2);
        }
        if (smax >= 0) {
            const long long m0 = (long long)n0, m1 = H0 * m0 + 2 * (long long)n1;
            const long long m2 = H0 * H0 * m0 + 4 * H0 * (long long)n1 + 4 * (long long)n2;
            int d = 0, dmin = 8, dmax = -8, t[8] = {8, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                d += 2 * ((p >> ((j & 1 ? 4 : 0) + (j >> 1))) & 1) - 1;
                dmin = min(dmin, d);
                dmax = max(dmax, d);
                int f = 1;
#pragma unroll
                for (int k = 1; k < 8; ++k) t[k] += (f *= d);
            }
            acc.s1 = 8 * m1 + t[1] * m0;
            acc.s2 = 8 * m2 + 2 * t[1] * m1 + t[2] * m0;
            acc.hmin = H0 + 2 * smin + dmin;
            acc.hmax = H0 + 2 * smax + dmax;
            const double M[8] = {(double)m0, (double)m1, (double)m2, m3, m4, m5, m6, m7};
            const double T[8] = {8.0,          (double)t[1], (double)t[2], (double)t[3],
                                 (double)t[4], (double)t[5], (double)t[6], (double)t[7]};
#pragma unroll
            for (int k = 3; k < 8; ++k) {
                double sum = 0.0;
                int binom = 1;
#pragma unroll
                for (int j = 0; j <= k; ++j) {
                    sum += (double)binom * T[j] * M[k - j];
                    binom = binom * (k - j) / (j + 1);
                }
                acc.s[k - 3] = sum;
            }
        }
    }
    // summed over all sites, sum h h' = sum u v + (mid - 128) sum v + (mid' - 128) sum h; the last term
    // is linear in s1, so every thread adds its share of it
    auto correlate = [&](Partial& p, long long uv, long long v) {
        p.cross = uv + (mid - 128) * v + (mid_s - 128) * p.s1;
        p.snap_s1 = v;  // less (128 - mid') per site, below
    };
    if (CORR) {
        correlate(acc, uv_sum, v_sum);
        acc.agree = agree;
    }
    __syncthreads();  // the counts have been read: their memory takes the values to add up
    long long* buf = reinterpret_cast<long long*>(hist);
    put_partial<NT>(acc, buf);
    if (__any_sync(0xffffffffu, far)) {
        Partial rest = empty_partial();
        longlong2 cross = make_longlong2(0, 0);
        const WalkGeom again = geom;
        walk_far<CORR>(again, &rest, &cross);
        if (CORR) correlate(rest, cross.x, cross.y);
        add_partial<NT>(rest, buf);
    }
    cta_reduce<NT>(buf, &partials[blockIdx.x]);
    if (threadIdx.x == 0) {
        __threadfence();  // the CTA's partial, ordered before this by the barrier
        last = atomicAdd(&ws->ticket, 1u) == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    static_assert(AN_MAX_GRID <= NT, "one partial per thread");
    acc = empty_partial();
    if (threadIdx.x < gridDim.x) {
        const longlong2* q = reinterpret_cast<const longlong2*>(partials + threadIdx.x);
        longlong2* d = reinterpret_cast<longlong2*>(&acc);
#pragma unroll
        for (int k = 0; k < (int)(sizeof(Partial) / 16); ++k) d[k] = __ldcg(q + k);
    }
    put_partial<NT>(acc, buf);
    cta_reduce<NT>(buf, out);
    if (CORR && threadIdx.x == 0) out->snap_s1 += (mid_s - 128) * (long long)(rows << lx);
}

// {Hs(y) - c, h(0, y) - c} of every row, from the row tables of the lattice measured last.
__global__ void __launch_bounds__(AN_ROW_THREADS)
row_heights_kernel(const int* __restrict__ rowinfo, const int64_t* __restrict__ rowstart, int lx, int ly, int64_t c,
                   const WalkState* __restrict__ ws, int2* __restrict__ out)
{
    __shared__ long long base_s[AN_MAX_BLOCKS];
    const uint64_t rows = 1ull << ly;
    const int lgb = row_block_lg(ly);
    row_block_bases<AN_ROW_THREADS>(ws->block[0], (int)(rows >> lgb), base_s);
    for (uint64_t y = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; y < rows; y += (uint64_t)gridDim.x * blockDim.x) {
        const int64_t h = rowstart[y] + base_s[y >> lgb] - c;
        out[y] = make_int2((int32_t)h, (int32_t)(h + row_sum(row_word(rowinfo, y, lx))));
    }
}

cudaError_t analysis_alloc(AnalysisScratch* s, int lx, int ly)
{
    const size_t rows = 1ull << ly;
    s->rows_cap = rows;
    cudaError_t e;
    // two row tables (system and snapshot) and partials, final record and the walk's state
    if ((e = cudaMalloc(&s->rowinfo, 2 * rows * row_ints(lx) * sizeof(int))) != cudaSuccess) return e;
    if ((e = cudaMalloc(&s->rowstart, 2 * rows * sizeof(int64_t))) != cudaSuccess) return e;
    const size_t acc = (AN_MAX_GRID + 1) * sizeof(Partial) + sizeof(WalkState);
    return cudaMalloc(&s->acc, acc);
}

void analysis_free(AnalysisScratch* s)
{
    cudaFree(s->rowinfo);
    cudaFree(s->rowstart);
    cudaFree(s->acc);
    s->rowinfo = nullptr;
    s->rowstart = nullptr;
    s->acc = nullptr;
}

size_t analysis_record_bytes() { return sizeof(Partial); }

void analysis_decode_record(const void* rec, MomentsOut* out)
{
    Partial h;
    memcpy(&h, rec, sizeof h);
    out->s1 = h.s1;
    out->s2 = h.s2;
    for (int k = 0; k < 5; ++k) out->s3to7[k] = h.s[k];
    out->hmin = h.hmin;
    out->hmax = h.hmax;
    out->cross = h.cross;
    out->agree = h.agree;
    out->snap_s1 = h.snap_s1;
}

static WalkState* walk_state(AnalysisScratch* s)
{
    return reinterpret_cast<WalkState*>(reinterpret_cast<Partial*>(s->acc) + AN_MAX_GRID + 1);
}

static void launch_rows(const uint32_t* d_sys, const uint32_t* d_snap, int lx, int ly, AnalysisScratch* s,
                        bool starts, cudaStream_t st)
{
    const dim3 grid(1u << (ly - row_block_lg(ly)), d_snap ? 2 : 1);
    auto kern = aligned16(d_sys) && aligned16(d_snap) ? row_kernel<false> : row_kernel<true>;
    kern<<<grid, AN_ROW_THREADS, 0, st>>>(d_sys, d_snap, lx, ly, s->rowinfo, starts ? s->rowstart : nullptr, walk_state(s));
}

cudaError_t analysis_moments_record(const uint32_t* d_sys, const uint32_t* d_snap, int lx, int ly,
                                    AnalysisScratch* s, void* d_rec, cudaStream_t st)
{
    launch_rows(d_sys, d_snap, lx, ly, s, true, st);
    // CTAs per row parity: a warp for each of their four schedulers as long as that is at most half
    // the SMs
    const uint64_t items = walk_items(lx, ly);
    const unsigned threads = walk_threads(d_snap != nullptr);
    const uint64_t want = (items + 3) / 4;
    const unsigned grid = 2 * (unsigned)(want < AN_MAX_GRID / 2 ? want : AN_MAX_GRID / 2);
    auto kern = d_snap ? walk_kernel<true> : walk_kernel<false>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, WALK_SMEM);
    if (e != cudaSuccess) return e;
    kern<<<grid, threads, WALK_SMEM, st>>>(d_sys, d_snap, lx, ly, s->rowinfo, s->rowstart,
                                           reinterpret_cast<Partial*>(s->acc), reinterpret_cast<Partial*>(d_rec),
                                           walk_state(s));
    return cudaGetLastError();
}

cudaError_t analysis_row_heights(AnalysisScratch* s, int lx, int ly, int64_t c, int2* d_out, cudaStream_t st)
{
    const uint64_t rows = 1ull << ly;
    const unsigned grid = (unsigned)(rows / AN_ROW_THREADS < 592 ? rows / AN_ROW_THREADS + 1 : 592);
    row_heights_kernel<<<grid, AN_ROW_THREADS, 0, st>>>(s->rowinfo, s->rowstart, lx, ly, c, walk_state(s), d_out);
    return cudaGetLastError();
}

cudaError_t analysis_moments(const uint32_t* d_sys, const uint32_t* d_snap, int lx, int ly,
                             AnalysisScratch* s, MomentsOut* out, cudaStream_t st)
{
    Partial* fin = reinterpret_cast<Partial*>(s->acc) + AN_MAX_GRID;
    cudaError_t e = analysis_moments_record(d_sys, d_snap, lx, ly, s, fin, st);
    if (e != cudaSuccess) return e;
    Partial h;
    if ((e = cudaMemcpyAsync(&h, fin, sizeof(Partial), cudaMemcpyDeviceToHost, st)) != cudaSuccess)
        return e;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
    analysis_decode_record(&h, out);
    return cudaSuccess;
}

// ---- invariants ----
// columns: thread per (x parity a, word column j, band of 256 rows); per-bit counters.
__global__ void colsum_kernel(const uint32_t* __restrict__ sys, int lx, int ly, int* colsum)
{
    const uint64_t Wr = 1ull << (lx - 6);
    const uint64_t Q = 1ull << (lx + ly - 6);
    const uint64_t rows = 1ull << ly;
    const uint64_t band = rows < 256 ? rows : 256;
    const uint64_t nb = rows / band;
    const uint64_t total = 2 * Wr * nb;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t j = i % Wr;
        const int a = (int)((i / Wr) & 1);
        const uint64_t b = i / (2 * Wr);
        int cnt[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) cnt[k] = 0;
        for (uint64_t y = b * band; y < (b + 1) * band; ++y) {
            const int sub = a ^ (int)(y & 1);
            const uint32_t w = sys[(sub ? 2 * Q : 0) + Q + y * Wr + j];
#pragma unroll
            for (int k = 0; k < 32; ++k) cnt[k] += (w >> k) & 1u;
        }
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            const uint64_t x = 64 * j + 2 * k + a;
            atomicAdd(&colsum[x], 2 * cnt[k] - (int)band);
        }
    }
}

__global__ void invariants_kernel(const uint32_t* __restrict__ sys, int lx, int ly,
                                  const int* __restrict__ rowinfo, const int* __restrict__ colsum,
                                  unsigned long long* rep)
{
    const uint64_t Wr = 1ull << (lx - 6);
    const uint64_t Q = 1ull << (lx + ly - 6);
    const uint64_t rows = 1ull << ly;
    const uint64_t L = 1ull << lx;
    unsigned long long badr = 0, badc = 0, badp = 0;
    const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t y = tid; y < rows; y += nth) badr += row_sum(row_word(rowinfo, y, lx)) != 0;
    for (uint64_t x = tid; x < L; x += nth) badc += colsum[x] != 0;
    // plaquettes: per (sublattice, row, word)
    for (uint64_t i = tid; i < 2 * Q; i += nth) {
        const int sub = (int)(i / Q);
        const uint64_t r = i % Q;
        const uint64_t y = r / Wr, j = r % Wr;
        const uint64_t bt = sub ? 2 * Q : 0, bo = sub ? 0 : 2 * Q;
        const int A = sub ^ (int)(y & 1);  // x parity of this sublattice in row y
        const uint32_t a = sys[bt + y * Wr + j];          // s_x(x,y)
        const uint32_t b = sys[bt + Q + y * Wr + j];      // s_y(x,y)
        uint32_t c;                                        // s_y(x-1,y)
        const uint32_t oy = sys[bo + Q + y * Wr + j];
        if (A) c = oy;
        else c = (oy << 1) | (sys[bo + Q + y * Wr + ((j + Wr - 1) & (Wr - 1))] >> 31);
        const uint32_t d = sys[bo + ((y + rows - 1) & (rows - 1)) * Wr + j];  // s_x(x,y-1)
        const uint32_t bad = ((a ^ c) ^ (b ^ d)) | ((a & c) ^ (b & d));
        badp += __popc(bad);
    }
    for (int o = 16; o > 0; o >>= 1) {
        badr += __shfl_xor_sync(0xffffffffu, badr, o);
        badc += __shfl_xor_sync(0xffffffffu, badc, o);
        badp += __shfl_xor_sync(0xffffffffu, badp, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&rep[0], badr);
        atomicAdd(&rep[1], badc);
        atomicAdd(&rep[2], badp);
    }
}

cudaError_t analysis_invariants(const uint32_t* d_sys, int lx, int ly, AnalysisScratch* s,
                                int64_t rep[3], cudaStream_t st)
{
    const uint64_t L = 1ull << lx;
    int* colsum = nullptr;
    cudaError_t e;
    if ((e = cudaMallocAsync(&colsum, L * sizeof(int) + 64, st)) != cudaSuccess) return e;
    unsigned long long* drep = reinterpret_cast<unsigned long long*>(colsum + L);
    cudaMemsetAsync(colsum, 0, L * sizeof(int) + 64, st);
    launch_rows(d_sys, nullptr, lx, ly, s, false, st);
    colsum_kernel<<<512, 256, 0, st>>>(d_sys, lx, ly, colsum);
    invariants_kernel<<<1184, 256, 0, st>>>(d_sys, lx, ly, s->rowinfo, colsum, drep);
    unsigned long long h[3] = {0, 0, 0};
    cudaMemcpyAsync(h, drep, sizeof(h), cudaMemcpyDeviceToHost, st);
    e = cudaStreamSynchronize(st);
    cudaFreeAsync(colsum, st);
    if (e == cudaSuccess) e = cudaGetLastError();
    rep[0] = (int64_t)h[0];
    rep[1] = (int64_t)h[1];
    rep[2] = (int64_t)h[2];
    return e;
}

}  // namespace kpzb

// ---------------------------------------------------------------------------------------
// Roughness without any allocation (kpzb_roughness_noalloc).
//
// Some callers cannot allocate device memory at the point where they want a measurement:
// an application whose memory manager owns the whole device (a caching allocator that must
// see every allocation, or a budget already spent on lattices), or a timing loop that must
// not stall other streams -- cudaMalloc and cudaFree can synchronize the device.  For them
// this entry point reads a caller's device lattice and writes the caller's host output, and
// keeps its scratch (row tables and per-CTA partial sums) in one file-scope device array of
// fixed size.  Every GPU that loads the library's module holds the array until the process
// exits.
//
// Limit: ly <= NOALLOC_MAX_LY (at most 65536 rows); any lx the other entry points accept.
// The array is shared by every call: concurrent calls that overlap on the GPU (on different
// streams or host threads) race on it and must be serialized by the caller.  Every kernel
// writes each scratch word before reading it, so nothing has to be cleared between calls.
// Set-up: the array's device address is looked up with cudaGetSymbolAddress once per device
// and CUDA context, while that device is current, and cached under the context's unique id;
// a context created anew (after the caller's cudaDeviceReset) gets a fresh lookup.  That
// first call may also load the library's module, and the array with it, so a caller with a
// window in which nothing may be allocated makes one call before the window opens; the
// first call on a device should come before any stream capture the caller starts.
// ---------------------------------------------------------------------------------------
namespace kpzb {

constexpr int NOALLOC_MAX_LY = 16;
constexpr size_t NOALLOC_ROWINFO = (1ull << NOALLOC_MAX_LY) * sizeof(int4);
constexpr size_t NOALLOC_ROWSTART = (1ull << NOALLOC_MAX_LY) * sizeof(int64_t);
constexpr size_t NOALLOC_PARTIALS = (AN_MAX_GRID + 1) * sizeof(Partial) + sizeof(WalkState);
constexpr size_t NOALLOC_BYTES = NOALLOC_ROWINFO + NOALLOC_ROWSTART + NOALLOC_PARTIALS;

static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_BYTES];

namespace {
// driver entry points for the current context and its process-unique id (CUDA >= 12.0),
// resolved once through the runtime so the library needs no link against libcuda
using CtxGetCurrentFn = int (*)(void**);
using CtxGetIdFn = int (*)(void*, unsigned long long*);
struct NoallocSetup {
    unsigned long long ctx_id = 0;
    void* addr = nullptr;
};
std::mutex g_noalloc_mu;
std::map<int, NoallocSetup> g_noalloc_setup;  // per device: context id -> symbol address
CtxGetCurrentFn g_ctx_get_current = nullptr;
CtxGetIdFn g_ctx_get_id = nullptr;
bool g_ctx_fns_looked_up = false;

// id of the context current on this thread; false when there is none (or it is gone)
bool current_ctx_id(unsigned long long* id)
{
    if (!g_ctx_fns_looked_up) {
        g_ctx_fns_looked_up = true;
        cudaDriverEntryPointQueryResult q1, q2;
        void* f1 = nullptr;
        void* f2 = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &q1) ==
                cudaSuccess && q1 == cudaDriverEntryPointSuccess &&
            cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &q2) == cudaSuccess &&
            q2 == cudaDriverEntryPointSuccess) {
            g_ctx_get_current = reinterpret_cast<CtxGetCurrentFn>(f1);
            g_ctx_get_id = reinterpret_cast<CtxGetIdFn>(f2);
        }
    }
    if (!g_ctx_get_current || !g_ctx_get_id) return false;
    void* ctx = nullptr;
    if (g_ctx_get_current(&ctx) != 0 || !ctx) return false;
    return g_ctx_get_id(ctx, id) == 0;
}
}  // namespace

// The scratch array's device address on the current device (set-up once per device and
// context; see above).
static cudaError_t noalloc_scratch_addr(int dev, void** out)
{
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    unsigned long long id = 0;
    const bool have_ctx = current_ctx_id(&id);
    auto it = g_noalloc_setup.find(dev);
    if (have_ctx && it != g_noalloc_setup.end() && it->second.ctx_id == id && it->second.addr) {
        *out = it->second.addr;
        return cudaSuccess;
    }
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    if (!p) return cudaErrorInvalidSymbol;
    unsigned long long id_after = 0;
    // the lookup makes the device's primary context current if none was
    if (current_ctx_id(&id_after)) g_noalloc_setup[dev] = NoallocSetup{id_after, p};
    else g_noalloc_setup.erase(dev);  // no id to key on: look up again next time
    *out = p;
    return cudaSuccess;
}

}  // namespace kpzb

extern "C" kpzb_status kpzb_roughness_noalloc(const uint32_t* d_cbbit, int lx, int ly, double out[8],
                                              void* stream)
{
    using namespace kpzb;
    if (!d_cbbit || !out) return fail(KPZB_EINVAL, "null lattice or output");
    if ((uintptr_t)d_cbbit & 3u) return fail(KPZB_EINVAL, "lattice not on a word boundary");
    if (lx < 8 || lx > 30 || ly < 2 || lx + ly < 14 || lx + ly > 38)
        return fail(KPZB_EINVAL, "lattice size out of range (8<=lx<=30, 14<=lx+ly<=38)");
    if (ly > NOALLOC_MAX_LY)
        return fail(KPZB_EINVAL, "ly > 16: the fixed no-allocation scratch holds at most 65536 rows");
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    void* addr = nullptr;
    e = noalloc_scratch_addr(dev, &addr);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(no-alloc scratch)");
    unsigned char* base = static_cast<unsigned char*>(addr);
    AnalysisScratch view;
    view.rowinfo = reinterpret_cast<int*>(base);
    view.rowstart = reinterpret_cast<int64_t*>(base + NOALLOC_ROWINFO);
    view.acc = reinterpret_cast<unsigned long long*>(base + NOALLOC_ROWINFO + NOALLOC_ROWSTART);
    view.rows_cap = 1ull << NOALLOC_MAX_LY;
    MomentsOut m;
    e = analysis_moments(d_cbbit, nullptr, lx, ly, &view, &m, static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return cuda_fail(e, "roughness (no-alloc)");
    const long double N = (long double)((uint64_t)1 << (lx + ly));
    long double h[7];
    h[0] = (long double)m.s1 / N;
    h[1] = (long double)m.s2 / N;
    for (int k = 0; k < 5; ++k) h[2 + k] = (long double)m.s3to7[k] / N;
    out[0] = (double)(h[1] - h[0] * h[0]);
    for (int k = 0; k < 7; ++k) out[1 + k] = (double)h[k];
    return KPZB_OK;
}

