// expand.cuh -- the sparse expansion with on-chip deduplication: the GPU
// form of Hybrid_solution's SPA loop (dim3.hpp:952-973).
//
// For an x row the candidates are every z of S row y for every y of R row x.
// Rows are binned by u = min(candidates, m), an upper bound on their distinct
// outputs:
//   class 1 (u <= cap_w):  one warp per row, a private shared-memory hash set
//   class 2 (u <= cap_b):  one CTA per row, a shared-memory hash set
//   class 3/4 (u > cap_b): one CTA per row, a shared-memory bitmap over one
//                          z tile at a time (S is bucketed by (y, z tile));
//                          class 4 (u > kHugeRow) rows are scheduled first.
// CTA classes take rows dynamically from an atomic counter.  The single pass
// (single.cuh, packed.cuh) expands each row once; ordered output (ordered.cuh)
// expands it twice, counting and then writing at exact offsets.
#pragma once
#include "common.cuh"
#include "items.h"

namespace dim3g {

constexpr uint32_t kEmpty32 = 0xFFFFFFFFu;
constexpr uint32_t kHugeRow = 1u << 16;
constexpr uint32_t kWarpWorkMax = 1u << 14;  // candidates a single warp takes alone
// Entries a single warp takes alone.  A hub's row may have next to no
// candidates and hundreds of thousands of entries to look up: 320K entries took
// a warp 3.9 ms, and a pack, which does more an entry, 5.3.
constexpr uint32_t kWarpEntries = 1024;
// Tiny rows (few distinct z, few candidates) are expanded many to a warp
// (packed.cuh).
constexpr uint32_t kTinyU = 256, kTinyW = 4096;

// A hash-class row dedups with a bitmap over the whole z domain instead of
// a hash set when that bitmap fits the kernel's table memory (2^slots_lg
// words) and holds at most kBitmapPerZ ids per distinct z (m <= 128 u, u =
// min(candidates, m)): no probing, one atomicOr per candidate, at m / 32
// words to clear against 2u to 4u.  (1.2M-edge 2-hop, m = 121K: block rows
// 983 us at 32 ids per distinct z, 677 at 128.)
constexpr uint64_t kBitmapPerZ = 128;
__device__ __forceinline__ bool use_row_bitmap(uint32_t m, uint32_t u, uint32_t slots_lg) {
    return (uint64_t)m <= (32ull << slots_lg) && (uint64_t)m <= kBitmapPerZ * u;
}
// Row class from its candidates w and u = min(w, m): 5 (one warp, small
// table; only where the caller runs that kernel) for tiny rows, 1 (one warp)
// for few distinct z and few candidates, 2 (one CTA, hash set or bitmap) up
// to cap_b distinct, 3 / 4 (one CTA, z-tile bitmaps; 4 = huge, scheduled
// first) beyond; 0 for an empty row.
__device__ __forceinline__ uint32_t row_class(unsigned long long w, uint32_t u, uint32_t ne, uint32_t cap_w,
                                              uint32_t cap_b, bool tiny) {
    if (u == 0) return 0;
    if (tiny && u <= kTinyU && w <= kTinyW && ne <= kWarpEntries) return 5;
    if (u <= cap_w && w <= kWarpWorkMax && ne <= kWarpEntries) return 1;
    if (u <= cap_b) return 2;
    return u <= kHugeRow ? 3 : 4;
}
// The block class's distinct bound for COUNT rows: larger rows are ranked over
// a bitmap (aggregate.cuh), which costs by the z domain where a map costs by
// its slots; below 128 z a distinct z the ranks are cheaper than the larger
// maps.  4000 rows, ranked and in maps: of 2500 distinct z, m = 173K 0.226 and
// 0.231 ms, m = 346K 0.325 and 0.222; of 5000, m = 173K 0.32 and 0.45, m = 346K
// 0.41 and 0.45, m = 691K 0.66 and 0.43.  (The 1M-tuple COUNT, m = 196K: 3.41
// ms, 3.57 with the bound at cap_b / 2, 4.49 with none.)
__host__ __device__ __forceinline__ uint32_t agg_cap_b(uint64_t m, uint32_t cap_b) {
    return m <= 128ull * (cap_b / 4) ? cap_b / 4 : (m <= 128ull * (cap_b / 2) ? cap_b / 2 : cap_b);
}
// Words of a whole-domain bitmap, rounded to uint4 and at least 32 (idle
// lanes of TileBitmap touch words 0..31).
__host__ __device__ __forceinline__ uint32_t row_bitmap_words(uint32_t m) {
    const uint32_t w = (((m + 31) >> 5) + 3) & ~3u;
    return w < 32 ? 32 : w;
}

struct RowCtx {
    const uint32_t* JR_R;  // n+1 row pointers of R by x id
    const uint32_t* IC_R;  // y ids
    const uint32_t* JR_S;  // k*T+1 row pointers of S by (y id, z tile)
    const uint32_t* IC_S;  // z ids
    const uint32_t* VS;    // z values, parallel to IC_S (value paths when ISV is nullptr)
    const uint2* ISV;      // (z id, z value) pairs parallel to IC_S, or nullptr (value paths load one pair)
    uint32_t T;            // z tiles
    uint32_t tile_width;   // z ids per tile (bitmap width)
    uint32_t m;            // z domain size
    uint32_t cta_rr;       // CTA rows' walk: 0 flattened, 1 chunks round-robin, 2 chunks split, 3 balanced (cta_expand)
    uint32_t flat_avg;     // cross-segment gather below this many candidates a segment (0: kFlatAvgMax)
    const uint32_t* ucap;  // per row min(candidates, m)
    uint32_t* cnt;         // per row distinct count (count pass output)
    const unsigned long long* off;  // per row output offset (write pass input)
    const uint32_t* id2x;
    const uint32_t* id2z;
    uint2* out;
    uint32_t* err;
    uint32_t* next_row;    // dynamic row counters of the CTA classes
};

// The z ids of S's entries, from the id array or from the (z id, z value)
// pairs (step 2).
struct ZIds {
    const uint32_t* a;
    uint32_t step;
    __device__ __forceinline__ uint32_t operator[](uint64_t j) const { return __ldg(&a[j * step]); }
};

__device__ __forceinline__ uint32_t ceil_log2(uint32_t v) { return v <= 1 ? 0 : 32 - __clz(v - 1); }

// Insert z into an open-addressing set of 2^lg 32-bit slots in shared memory.
// Returns true for the first insertion of z.
__device__ __forceinline__ bool smem_set_insert(uint32_t* tab, uint32_t lg, uint32_t z, uint32_t* err) {
    const uint32_t mask = (1u << lg) - 1;
    uint32_t h = (z * 0x9E3779B1u) >> (32 - lg);
    volatile uint32_t* vt = tab;
    for (uint32_t p = 0; p <= mask; p++) {
        uint32_t cur = vt[h];
        if (cur == z) return false;
        if (cur == kEmpty32) {
            uint32_t prev = atomicCAS(&tab[h], kEmpty32, z);
            if (prev == kEmpty32) return true;
            if (prev == z) return false;
        }
        h = (h + 1) & mask;
    }
    raise_error(err, kErrTableFull);
    return false;
}

#ifndef DIM3G_UNROLL
#define DIM3G_UNROLL 4
#endif
#ifndef DIM3G_MIN_PIECE
#define DIM3G_MIN_PIECE 256
#endif
#ifndef DIM3G_FLAT_AVG
#define DIM3G_FLAT_AVG 96
#endif
constexpr uint32_t kUnroll = DIM3G_UNROLL;
constexpr uint32_t kMinPiece = DIM3G_MIN_PIECE;
// A chunk whose segments average fewer candidates than this is gathered
// across segment boundaries (see warp_expand); RowCtx::flat_avg overrides it
// per launch (the single pass sets it per row class).
constexpr uint32_t kFlatAvgMax = DIM3G_FLAT_AVG;

// Warp-level expansion of the candidates of R entries [e0, e1) over S tiles
// [t0, t1).  Entries are taken 32 at a time; a warp prefix sum over their S
// segment lengths flattens the chunk's candidates into [0, total), which is
// cut into a power-of-two number (<= nparts) of contiguous pieces of at least
// kMinPiece candidates; the calling warp takes piece `part`.  When the
// chunk's segments are short on average it gathers its piece across segment
// boundaries (each lane looks up its candidate's segment); otherwise it
// finds the segment holding its first candidate with one ballot over the
// lanes' inclusive prefixes, then walks the segments overlapping its piece,
// the lanes striding each segment kUnroll x 32 candidates at a time.
//   set.insert(z, active) -> bool   per lane (false when !active)
//   sink.take(b[], v[])             warp-collective once per group: b[u] is
//                                   the ballot of first insertions of step u;
//                                   v[u] is the lane's z value when the sink
//                                   asks for values (Sink::kValues), loaded
//                                   together with the z id to hide latency
// One 32-entry chunk of R entries: per lane its S segment over tiles
// [t0, t1) (start, length), the warp's inclusive / exclusive prefixes of the
// lengths and the chunk's candidate total.
struct Chunk {
    uint32_t s0, len, incl, excl, total;
};

__device__ __forceinline__ Chunk load_chunk(const RowCtx& c, uint32_t eb, uint32_t e1, uint32_t t0, uint32_t t1,
                                            uint64_t pol) {
    Chunk ch;
    const uint32_t e = eb + lane_id();
    ch.s0 = 0;
    ch.len = 0;
    if (e < e1) {
        const uint32_t y = ld_keep(&c.IC_R[e], pol);
        const uint64_t r = (uint64_t)y * c.T;
        ch.s0 = ld_keep(&c.JR_S[r + t0], pol);
        ch.len = ld_keep(&c.JR_S[r + t1], pol) - ch.s0;
    }
    ch.incl = warp_incl_scan(ch.len);
    if (__any_sync(0xffffffffu, ch.incl < ch.len)) raise_error(c.err, kErrCountRange);
    ch.total = __shfl_sync(0xffffffffu, ch.incl, 31);
    ch.excl = ch.incl - ch.len;
    return ch;
}

// Candidates [p0, p1) of a chunk through the set into the sink (the calling
// warp).  Many short segments: gather across segment boundaries -- each lane
// finds the segment of its candidate (the number of lanes with incl <= c;
// incl is nondecreasing over lanes) by a 5-step binary search over the
// lanes' prefixes, so one group of kUnroll x 32 loads covers many segments
// with a single memory latency.  Long segments: the lanes stride each
// segment overlapping the piece, kUnroll x 32 candidates at a time, all
// loads of a group issued first.
// One candidate's z id (and z value when the sink asks for values): a pair
// load from ISV, or the id and value arrays.
template <bool kPair, bool kValues>
__device__ __forceinline__ void load_cand(const RowCtx& c, uint32_t j, bool act, uint64_t pol, uint32_t& z,
                                          uint32_t& v) {
    if (kPair && kValues) {
        const uint2 p = act ? ld_keep2(&c.ISV[j], pol) : make_uint2(kEmpty32, 0u);
        z = p.x;
        v = p.y;
    } else {
        z = act ? ld_keep(&c.IC_S[j], pol) : kEmpty32;
        if (kValues) v = act ? ld_keep(&c.VS[j], pol) : 0u;
    }
}

template <bool kPair, class Set, class Sink>
__device__ __forceinline__ void expand_piece_impl(const RowCtx& c, const Chunk& ch, uint32_t p0, uint32_t p1,
                                                  Set& set, Sink& sink, uint64_t pol) {
    const uint32_t lane = lane_id();
    const uint32_t nseg = __popc(__ballot_sync(0xffffffffu, ch.len != 0));
    if (ch.total < (c.flat_avg ? c.flat_avg : kFlatAvgMax) * nseg) {
        for (uint32_t cb = p0; cb < p1; cb += 32 * kUnroll) {
            uint32_t z[kUnroll], v[kUnroll];
#pragma unroll
            for (uint32_t u = 0; u < kUnroll; u++) {
                const uint32_t cc = cb + u * 32 + lane;
                const bool act = cc < p1;
                const uint32_t ci = act ? cc : p0;  // idle lanes search a valid index
                uint32_t k = 0;
#pragma unroll
                for (uint32_t step = 16; step >= 1; step >>= 1)
                    if (__shfl_sync(0xffffffffu, ch.incl, k + step - 1) <= ci) k += step;
                const uint32_t j = __shfl_sync(0xffffffffu, ch.s0, k) + (ci - __shfl_sync(0xffffffffu, ch.excl, k));
                load_cand<kPair, Sink::kValues>(c, j, act, pol, z[u], v[u]);
            }
            uint32_t b[kUnroll];
#pragma unroll
            for (uint32_t u = 0; u < kUnroll; u++)
                b[u] = (cb + u * 32 < p1) ? __ballot_sync(0xffffffffu, set.insert(z[u], z[u] != kEmpty32)) : 0u;
            sink.take(b, v);
        }
        return;
    }
    // first segment holding candidate p0: lanes with incl <= p0 form a prefix
    for (uint32_t k = __popc(__ballot_sync(0xffffffffu, ch.incl <= p0)); k < 32; k++) {
        const uint32_t kex = __shfl_sync(0xffffffffu, ch.excl, k);
        if (kex >= p1) break;
        const uint32_t klen = __shfl_sync(0xffffffffu, ch.len, k);
        const uint32_t ks0 = __shfl_sync(0xffffffffu, ch.s0, k);
        const uint32_t lo = (p0 > kex ? p0 - kex : 0);
        const uint32_t hi = (kex + klen < p1 ? klen : p1 - kex);
        uint32_t jb = lo;
        // full groups: kUnroll x 32 candidates, all loads issued first
        for (; jb + 32 * kUnroll <= hi; jb += 32 * kUnroll) {
            uint32_t z[kUnroll], v[kUnroll];
#pragma unroll
            for (uint32_t u = 0; u < kUnroll; u++) load_cand<kPair, Sink::kValues>(c, ks0 + jb + u * 32 + lane, true, pol, z[u], v[u]);
            uint32_t b[kUnroll];
#pragma unroll
            for (uint32_t u = 0; u < kUnroll; u++) b[u] = __ballot_sync(0xffffffffu, set.insert(z[u], true));
            sink.take(b, v);
        }
        // tail (< kUnroll x 32 left): all its loads issued together, so one
        // load latency per segment tail; steps past the end are skipped
        // warp-uniformly
        if (jb < hi) {
            uint32_t z[kUnroll], v[kUnroll];
#pragma unroll
            for (uint32_t u = 0; u < kUnroll; u++) {
                const uint32_t j = jb + u * 32 + lane;
                load_cand<kPair, Sink::kValues>(c, ks0 + j, j < hi, pol, z[u], v[u]);
            }
            uint32_t b[kUnroll];
#pragma unroll
            for (uint32_t u = 0; u < kUnroll; u++)
                b[u] = (jb + u * 32 < hi) ? __ballot_sync(0xffffffffu, set.insert(z[u], z[u] != kEmpty32)) : 0u;
            sink.take(b, v);
        }
    }
}

// Candidates [p0, p1) of a chunk: paired loads where the (z id, z value)
// pairs exist and the sink takes values.
template <class Set, class Sink>
__device__ __forceinline__ void expand_piece(const RowCtx& c, const Chunk& ch, uint32_t p0, uint32_t p1, Set& set,
                                             Sink& sink, uint64_t pol) {
    if (Sink::kValues && c.ISV != nullptr)
        expand_piece_impl<true>(c, ch, p0, p1, set, sink, pol);
    else
        expand_piece_impl<false>(c, ch, p0, p1, set, sink, pol);
}

// Warp-level expansion of the candidates of R entries [e0, e1) over S tiles
// [t0, t1).  Entries are taken 32 at a time; a warp prefix sum over their S
// segment lengths flattens the chunk's candidates into [0, total), which is
// cut into a power-of-two number (<= 2^nparts_lg) of contiguous pieces of at
// least kMinPiece candidates; the calling warp takes piece `part`.
//   set.insert(z, active) -> bool   per lane (false when !active)
//   sink.take(b[], v[])             warp-collective once per group: b[u] is
//                                   the ballot of first insertions of step u;
//                                   v[u] is the lane's z value when the sink
//                                   asks for values (Sink::kValues), loaded
//                                   together with the z id to hide latency
template <class Set, class Sink>
__device__ __forceinline__ void warp_expand(const RowCtx& c, uint32_t e0, uint32_t e1, uint32_t part,
                                            uint32_t nparts_lg, uint32_t t0, uint32_t t1, Set& set, Sink& sink) {
    const uint64_t pol = l2_keep_policy();
    for (uint32_t eb = e0; eb < e1; eb += 32) {
        const Chunk ch = load_chunk(c, eb, e1, t0, t1, pol);
        const uint32_t want = ch.total / kMinPiece;
        uint32_t np_lg = want <= 1 ? 0 : 31 - __clz(want);
        np_lg = np_lg > nparts_lg ? nparts_lg : np_lg;
        if (part >= (1u << np_lg)) continue;
        const uint32_t piece = (ch.total >> np_lg) + ((ch.total & ((1u << np_lg) - 1)) ? 1u : 0u);
        const uint32_t p0 = min(part * piece, ch.total);
        const uint32_t p1 = min(p0 + piece, ch.total);
        if (p0 < p1) expand_piece(c, ch, p0, p1, set, sink, pol);
    }
}

// Chunks a CTA defers to its cooperative phase (round-robin walk), and the
// staged segment table of the row-flattened and balanced walks (see
// cta_expand).
constexpr uint32_t kBigChunk = 4096, kBigCap = 64;
constexpr uint32_t kRowBlk = 1024;  // R entries staged at a time by the flattened / balanced walks
struct CtaChunks {
    uint32_t n;              // deferred chunks (may exceed kBigCap: the rest ran at once)
    uint32_t eb[kBigCap];
    union {
        struct {
            uint32_t s0[kRowBlk];    // segment start of each staged entry
            uint32_t incl[kRowBlk];  // flattened walk: inclusive prefix of the lengths; balanced walk: the lengths
        } seg;
        uint32_t bnd[2 * kRowBlk];   // a row's entries' S row bounds over all z tiles (bitmap rows)
    } st;
    uint32_t ctot[kRowBlk / 32];  // balanced walk: candidates of each staged 32-entry chunk
};

// Row-flattened CTA walk over R entries [e0, e1) and S tiles [t0, t1): the
// CTA stages kRowBlk entries' segment bounds in shared memory at once (one
// load latency for the whole block instead of one per 32-entry chunk),
// scans their lengths CTA-wide and splits the block's candidates evenly
// over the warps; each lane finds its candidate's segment by binary search
// in the staged prefixes.  Contains barriers; called by the whole CTA.
template <class Set, class Sink>
__device__ __forceinline__ void cta_expand_flat(const RowCtx& c, uint32_t e0, uint32_t e1, uint32_t t0, uint32_t t1,
                                                Set& set, Sink& sink, CtaChunks* cc) {
    const uint32_t tid = threadIdx.x, lane = lane_id(), wib = tid >> 5, nw = blockDim.x >> 5;
    const uint32_t per = (kRowBlk + blockDim.x - 1) / blockDim.x;  // entries per thread (<= 4)
    const uint64_t pol = l2_keep_policy();
    __shared__ uint32_t sm_scan[1024 / 32 + 1];
    for (uint32_t eb = e0; eb < e1; eb += kRowBlk) {
        const uint32_t ne = min(kRowBlk, e1 - eb);
        // stage: thread tid owns entries [tid*per, tid*per + per)
        uint32_t s0[4], len[4], sum = 0;
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) {
            s0[k] = 0;
            len[k] = 0;
            const uint32_t i = tid * per + k;
            if (k < per && i < ne) {
                const uint32_t y = ld_keep(&c.IC_R[eb + i], pol);
                const uint64_t r = (uint64_t)y * c.T;
                s0[k] = ld_keep(&c.JR_S[r + t0], pol);
                len[k] = ld_keep(&c.JR_S[r + t1], pol) - s0[k];
                sum += len[k];
            }
        }
        // CTA-wide exclusive scan of the threads' sums (blockDim <= 1024)
        const uint32_t inc = warp_incl_scan(sum);
        if (lane == 31) sm_scan[wib] = inc;
        __syncthreads();
        if (wib == 0) {
            const uint32_t v = lane < nw ? sm_scan[lane] : 0u;
            const uint32_t vi = warp_incl_scan(v);
            if (lane < nw) sm_scan[lane] = vi - v;
            if (lane == nw - 1) sm_scan[nw] = vi;
        }
        __syncthreads();
        uint32_t run = sm_scan[wib] + inc - sum;
        if (sm_scan[nw] < run) raise_error(c.err, kErrCountRange);  // 32-bit prefix wrapped
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) {
            const uint32_t i = tid * per + k;
            if (k < per && i < ne) {
                run += len[k];
                cc->st.seg.s0[i] = s0[k];
                cc->st.seg.incl[i] = run;
            }
        }
        const uint32_t total = sm_scan[nw];
        __syncthreads();
        // the warps' even shares of the block's candidates
        const uint32_t piece = (total + nw - 1) / nw;
        const uint32_t p0 = min(wib * piece, total), p1 = min(p0 + piece, total);
        for (uint32_t cb = p0; cb < p1; cb += 32 * kUnroll) {
            uint32_t z[kUnroll], v[kUnroll];
#pragma unroll
            for (uint32_t u = 0; u < kUnroll; u++) {
                const uint32_t ci = cb + u * 32 + lane;
                const bool act = ci < p1;
                // first staged entry with incl > ci
                uint32_t lo = 0, hi = ne - 1;
                while (lo < hi) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (cc->st.seg.incl[mid] > ci) hi = mid;
                    else lo = mid + 1;
                }
                const uint32_t excl = lo ? cc->st.seg.incl[lo - 1] : 0u;
                const uint32_t j = cc->st.seg.s0[lo] + (ci - excl);
                if (Sink::kValues && c.ISV != nullptr)
                    load_cand<true, true>(c, j, act, pol, z[u], v[u]);
                else
                    load_cand<false, Sink::kValues>(c, j, act, pol, z[u], v[u]);
            }
            uint32_t b[kUnroll];
#pragma unroll
            for (uint32_t u = 0; u < kUnroll; u++)
                b[u] = (cb + u * 32 < p1) ? __ballot_sync(0xffffffffu, set.insert(z[u], z[u] != kEmpty32)) : 0u;
            sink.take(b, v);
        }
        __syncthreads();  // the staged table is rewritten by the next block
    }
}

// Balanced walk, staging half: the warps stage the segments of R entries
// [eb, eb + ne) (ne <= kRowBlk) over S tiles [t0, t1) in shared memory, each
// warp loading whole 32-entry chunks (every entry is loaded once), with each
// chunk's candidate total.  No barrier; the expanding half follows one.
// (wib, nw): this warp's index among the nw warps that share the work.
__device__ __forceinline__ void balanced_stage(const RowCtx& c, uint32_t eb, uint32_t ne, uint32_t t0, uint32_t t1,
                                               CtaChunks* cc, uint64_t pol, uint32_t wib, uint32_t nw) {
    const uint32_t lane = lane_id();
    const uint32_t nch = (ne + 31) >> 5;
    for (uint32_t k = wib; k < nch; k += nw) {
        const uint32_t i = k * 32 + lane, e = eb + i;
        uint32_t s0 = 0, len = 0;
        if (i < ne) {
            const uint32_t y = ld_keep(&c.IC_R[e], pol);
            const uint64_t r = (uint64_t)y * c.T;
            s0 = ld_keep(&c.JR_S[r + t0], pol);
            len = ld_keep(&c.JR_S[r + t1], pol) - s0;
        }
        cc->st.seg.s0[i] = s0;
        cc->st.seg.incl[i] = len;
        const uint32_t inc = warp_incl_scan(len);
        if (__any_sync(0xffffffffu, inc < len)) raise_error(c.err, kErrCountRange);  // 32-bit prefix wrapped
        if (lane == 31) cc->ctot[k] = inc;
    }
}

// Balanced walk, expanding half: every warp takes an equal share of the
// staged block's candidates -- the chunks overlapping its share, each through
// expand_piece with the chunk rebuilt from shared memory -- so no warp idles
// at the next barrier while another expands a long chunk alone.  No barrier.
// s0 / len / ctot: the staged segment starts and lengths and the chunk
// totals (a CtaChunks' arrays, or a prefetched row's).
// dyn (optional, zeroed before the barrier that precedes this): a shared
// counter of pieces of dyn_piece candidates, which the warps take instead of
// equal static shares.
// dyn_piece 0: a warp's share of the candidates, at least 256 and at most
// this many (direct COUNT rows, whose tiles hold 4K candidates and up: a slice
// of the 16M-tuple COUNT takes 1024 ms in pieces of 256, 698 up to 1024, 646
// up to 4096).
constexpr uint32_t kDynPieceMax = 4096;
template <class Set, class Sink>
__device__ __forceinline__ void balanced_expand(const RowCtx& c, uint32_t ne, Set& set, Sink& sink,
                                                const uint32_t* s0a, const uint32_t* lena, const uint32_t* ctota,
                                                uint64_t pol, uint32_t wib, uint32_t nw, uint32_t* dyn = nullptr,
                                                uint32_t dyn_piece = 0) {
    const uint32_t lane = lane_id();
    const uint32_t nch = (ne + 31) >> 5;
    // prefix of the chunk totals (every warp computes it; nch <= 32)
    const uint32_t v = lane < nch ? ctota[lane] : 0u;
    const uint32_t inc = warp_incl_scan(v);
    if (__any_sync(0xffffffffu, inc < v)) raise_error(c.err, kErrCountRange);
    const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
    const uint32_t share = total / nw + (total % nw ? 1u : 0u);
    const Pieces pieces(dyn_piece ? dyn_piece : min(max((share + 127) & ~127u, 256u), kDynPieceMax), total);
    for (uint32_t round = 0;; round++) {
    uint32_t p0, p1;
    if (dyn) {
        uint32_t k0 = 0;
        if (lane == 0) k0 = atomicAdd(dyn, 1u);
        k0 = __shfl_sync(0xffffffffu, k0, 0);
        if (!pieces.at(k0, &p0, &p1)) break;
    } else if (round || !share_of(wib, nw, total, &p0, &p1)) {
        break;
    }
    // first chunk holding candidate p0: chunks with incl <= p0 form a prefix
    for (uint32_t k = __popc(__ballot_sync(0xffffffffu, lane < nch && inc <= p0)); k < nch; k++) {
        const uint32_t cin = __shfl_sync(0xffffffffu, inc, k), ctot = __shfl_sync(0xffffffffu, v, k);
        const uint32_t cex = cin - ctot;
        if (cex >= p1) break;
        if (ctot == 0) continue;
        Chunk ch;
        ch.s0 = s0a[k * 32 + lane];
        ch.len = lena[k * 32 + lane];
        ch.incl = warp_incl_scan(ch.len);
        ch.excl = ch.incl - ch.len;
        ch.total = ctot;
        const uint32_t lo = p0 > cex ? p0 - cex : 0u, hi = p1 < cin ? p1 - cex : ctot;
        expand_piece(c, ch, lo, hi, set, sink, pol);
    }
    }
}

// Balanced CTA walk over R entries [e0, e1) and S tiles [t0, t1), kRowBlk
// entries at a time.  Contains barriers; called by the whole CTA.
template <class Set, class Sink>
__device__ __forceinline__ void cta_expand_balanced(const RowCtx& c, uint32_t e0, uint32_t e1, uint32_t t0,
                                                    uint32_t t1, Set& set, Sink& sink, CtaChunks* cc) {
    const uint64_t pol = l2_keep_policy();
    const uint32_t wib = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (uint32_t eb = e0; eb < e1; eb += kRowBlk) {
        const uint32_t ne = min(kRowBlk, e1 - eb);
        balanced_stage(c, eb, ne, t0, t1, cc, pol, wib, nw);
        __syncthreads();
        balanced_expand(c, ne, set, sink, cc->st.seg.s0, cc->st.seg.incl, cc->ctot, pol, wib, nw);
        __syncthreads();  // the staged table is rewritten by the next block
    }
}

// CTA-level expansion of R entries [e0, e1) over S tiles [t0, t1), called
// by all warps of the CTA (2^nw_lg of them) with the same arguments.
// c.cta_rr selects the walk: 3 the balanced walk (cta_expand_balanced),
// 0 the row-flattened walk (cta_expand_flat),
// 2 every chunk split across the warps (warp_expand), 1 with at least as
// many chunks as warps, each warp takes whole
// chunks round-robin -- a chunk's entries and segment bounds are loaded by
// one warp, not by every warp -- and chunks of more than kBigChunk
// candidates are deferred and then split across all warps.  Otherwise every
// chunk is split across the warps (warp_expand).  Which is faster depends on
// the workload (the autotuner times both).  cc->n must be 0
// on entry (it is 0 again on return); contains barriers.
template <class Set, class Sink>
__device__ __forceinline__ void cta_expand(const RowCtx& c, uint32_t e0, uint32_t e1, uint32_t wib, uint32_t nw_lg,
                                           uint32_t t0, uint32_t t1, Set& set, Sink& sink, CtaChunks* cc) {
    const uint32_t nchunks = (e1 - e0 + 31) >> 5;
    if (c.cta_rr == 3) {
        cta_expand_balanced(c, e0, e1, t0, t1, set, sink, cc);
        return;
    }
    if (c.cta_rr == 0) {
        cta_expand_flat(c, e0, e1, t0, t1, set, sink, cc);
        return;
    }
    if (c.cta_rr == 2 || nchunks < (1u << nw_lg)) {
        warp_expand(c, e0, e1, wib, nw_lg, t0, t1, set, sink);
        return;
    }
    const uint64_t pol = l2_keep_policy();
    for (uint32_t ci = wib; ci < nchunks; ci += 1u << nw_lg) {
        const uint32_t eb = e0 + 32 * ci;
        const Chunk ch = load_chunk(c, eb, e1, t0, t1, pol);
        if (ch.total > kBigChunk) {
            uint32_t slot = 0;
            if (lane_id() == 0) slot = atomicAdd(&cc->n, 1u);
            slot = __shfl_sync(0xffffffffu, slot, 0);
            if (slot < kBigCap) {
                if (lane_id() == 0) cc->eb[slot] = eb;
                continue;
            }
        }
        if (ch.total) expand_piece(c, ch, 0, ch.total, set, sink, pol);
    }
    __syncthreads();
    const uint32_t nbig = min(cc->n, kBigCap);
    for (uint32_t i = 0; i < nbig; i++) {
        const uint32_t eb = cc->eb[i];
        warp_expand(c, eb, min(eb + 32, e1), wib, nw_lg, t0, t1, set, sink);
    }
    __syncthreads();
    if (threadIdx.x == 0) cc->n = 0;
}

// ----------------------------------------------------------------- sets
struct HashSet {
    uint32_t* tab;
    uint32_t lg;
    uint32_t* err;
    __device__ __forceinline__ bool insert(uint32_t z, bool act) { return act ? smem_set_insert(tab, lg, z, err) : false; }
};

// Bitmap over one z tile; branch-free (idle lanes OR a zero into words
// 0..31, so the bitmap allocation is at least 32 words).
struct TileBitmap {
    uint32_t* bm;
    uint32_t lo;
    __device__ __forceinline__ bool insert(uint32_t z, bool act) {
        const uint32_t zl = z - lo;
        const uint32_t w = act ? (zl >> 5) : lane_id();
        const uint32_t bit = act ? (1u << (zl & 31)) : 0u;
        return (atomicOr(&bm[w], bit) & bit) == 0 && act;
    }
};

// ---------------------------------------------------------------- sinks
struct CountSink {
    static constexpr bool kValues = false;
    uint32_t count = 0;
    template <uint32_t N>
    __device__ __forceinline__ void take(const uint32_t (&b)[N], const uint32_t (&)[N]) {
#pragma unroll
        for (uint32_t u = 0; u < N; u++) count += __popc(b[u]);
    }
};

// Emits first insertions at base + a row-local slot.  shared_pos == nullptr:
// the warp owns the row and counts locally; otherwise one shared-memory claim
// per group reserves the slots.
struct WriteSink {
    static constexpr bool kValues = true;
    uint2* out;
    uint32_t* err;
    unsigned long long base;
    uint32_t lim, xv;
    uint32_t* shared_pos;
    uint32_t local = 0;
    template <uint32_t N>
    __device__ __forceinline__ void take(const uint32_t (&b)[N], const uint32_t (&v)[N]) {
        uint32_t n = 0;
#pragma unroll
        for (uint32_t u = 0; u < N; u++) n += __popc(b[u]);
        if (n == 0) return;
        uint32_t pb;
        if (shared_pos) {
            pb = 0;
            if (lane_id() == 0) pb = atomicAdd(shared_pos, n);
            pb = __shfl_sync(0xffffffffu, pb, 0);
        } else {
            pb = local;
            local += n;
        }
        const uint32_t lt = lanemask_lt();
#pragma unroll
        for (uint32_t u = 0; u < N; u++) {
            if (b[u] & (1u << lane_id())) {
                const uint32_t pos = pb + __popc(b[u] & lt);
                if (pos < lim) st_stream(&out[base + pos], make_uint2(xv, v[u]));
                else raise_error(err, kErrOutputBound);
            }
            pb += __popc(b[u]);
        }
    }
};

// Next row of a CTA class, taken dynamically (the whole CTA gets the index).
__device__ __forceinline__ uint32_t cta_next_row(uint32_t* counter, uint32_t* s_row) {
    __syncthreads();
    if (threadIdx.x == 0) *s_row = atomicAdd(counter, 1u);
    __syncthreads();
    return *s_row;
}

// The rows' lists.  A row's bucket: 0 warp class; 1..3 block class, by
// distinct bound u <= cap_s, u <= cap_m, larger where the launches are split
// by hash-set size (else all 1); 4 huge and 5 other bitmap rows; 6 tiny rows;
// kRowBuckets none.
constexpr uint32_t kRowBuckets = 7;
struct RowBuckets {
    uint32_t cap_w, cap_b;  // row_class bounds
    bool tiny, split;
    uint32_t cap_s, cap_m;
    __device__ __forceinline__ uint32_t of(uint32_t cls, uint32_t u) const {
        if (cls == 1) return 0;
        if (cls == 2) return !split || u <= cap_s ? 1u : (u <= cap_m ? 2u : 3u);
        return cls == 0 ? kRowBuckets : (cls == 4 ? 4u : (cls == 3 ? 5u : 6u));
    }
};

// Per-row candidate count w = sum over y in R_x of |S_y|, u = min(w, m) and
// the row class (0: empty, or outside sel's A-tiles).  With check_range set
// (join-aggregate, 32-bit per-group counters) a row of 2^32 or more
// candidates raises kErrCountRange.
//
// A row's entries are a chain of dependent loads (row bounds, y id, S bounds),
// so the rows in flight bound the time: 2^lg lanes take a row, about as many
// as a row has entries on average (row_work_lanes), and a row of more than
// 4 x 2^lg entries is finished by its whole warp.  A warp for every row took
// 281 us for 1M rows of 10 entries.  Rows of more than kLongRow entries are
// left to the whole CTA at its end, kLongRows of them (where there are more,
// their warps do them side by side): a hub of 2M entries among 4M tuples held
// one warp, and the GPU with it -- the whole join 29.5 ms, 19.7 with the CTA;
// 20M-edge and 10M uniform joins the same either way.  The sums and the rows per bucket are
// added up per CTA in shared memory, then one atomic a CTA and counter.
constexpr uint32_t kLongRow = 2048, kLongRows = 4;
static __global__ void __launch_bounds__(256) k_row_work(RowCtx c, uint32_t n, uint32_t lg, RowBuckets rb,
                                                         bool check_range, SumAcc sel, uint32_t* __restrict__ ucap,
                                                         uint8_t* __restrict__ bucket, unsigned long long* outj,
                                                         unsigned long long* outj_cls, unsigned long long* nbucket) {
    __shared__ unsigned long long s_acc[6];
    __shared__ uint32_t s_n[kRowBuckets + 1];
    __shared__ uint32_t s_nlong;
    __shared__ uint3 s_long[kLongRows];  // row, its entries
    __shared__ unsigned long long s_w[kLongRows];
    if (threadIdx.x < 6) s_acc[threadIdx.x] = 0;
    if (threadIdx.x <= kRowBuckets) s_n[threadIdx.x] = 0;
    if (threadIdx.x < kLongRows) s_w[threadIdx.x] = 0;
    if (threadIdx.x == 0) s_nlong = 0;
    __syncthreads();
    auto candidates = [&](uint32_t e) {
        const uint64_t r = (uint64_t)__ldg(&c.IC_R[e]) * c.T;
        return __ldg(&c.JR_S[r + c.T]) - __ldg(&c.JR_S[r]);
    };
    auto finish = [&](uint64_t x, uint32_t ne, unsigned long long w) {
        const uint32_t u = (uint32_t)(w < c.m ? w : c.m);
        const uint32_t k = row_class(w, u, ne, rb.cap_w, rb.cap_b, rb.tiny), q = rb.of(k, u);
        ucap[x] = u;
        bucket[x] = (uint8_t)q;
        atomicAdd(&s_n[q], 1u);
        if (check_range && w >= 0xFFFFFFFFull) raise_error(c.err, kErrCountRange);
        if (w) {
            atomicAdd(&s_acc[0], w);
            atomicAdd(&s_acc[k], w);
        }
    };
    const uint32_t lane = lane_id(), G = 1u << lg, gl = lane & (G - 1), per = 32 >> lg;
    const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t x0 = gw * per; x0 < n; x0 += nwarps * per) {
        const uint64_t x = x0 + (lane >> lg);
        uint32_t e0 = 0, e1 = 0;
        const bool live = x < n && !(sel.tiles && !sel.selected(c.id2x[x]));  // summaries over a slice of A-tiles
        if (live) {
            e0 = c.JR_R[x];
            e1 = c.JR_R[x + 1];
        }
        const uint32_t ne = e1 - e0;
        bool later = ne > kLongRow;
        if (__any_sync(0xffffffffu, later)) {
            uint32_t slot = 0;
            if (later && gl == 0) slot = atomicAdd(&s_nlong, 1u);
            slot = __shfl_sync(0xffffffffu, slot, lane & ~(G - 1));
            later = later && slot < kLongRows;
            if (later && gl == 0) s_long[slot] = make_uint3((uint32_t)x, e0, e1);
            if (later) e1 = e0;
        }
        unsigned long long w = 0;
        const uint32_t head = e0 + min(e1 - e0, 4 * G);
        uint32_t y[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) y[k] = e0 + gl + k * G < head ? __ldg(&c.IC_R[e0 + gl + k * G]) : kEmpty32;
#pragma unroll
        for (uint32_t k = 0; k < 4; k++)
            if (y[k] != kEmpty32) {
                const uint64_t r = (uint64_t)y[k] * c.T;
                w += __ldg(&c.JR_S[r + c.T]) - __ldg(&c.JR_S[r]);
            }
        // the rest of the warp's long rows, all lanes on one row at a time
        for (uint32_t longs = __ballot_sync(0xffffffffu, gl == 0 && head < e1); longs; longs &= longs - 1) {
            const int src = __ffs(longs) - 1;
            const uint32_t b = __shfl_sync(0xffffffffu, head, src), e = __shfl_sync(0xffffffffu, e1, src);
            unsigned long long v = 0;
#pragma unroll 4
            for (uint32_t k = b + lane; k < e; k += 32) v += candidates(k);
            v = warp_sum(v);
            if ((int)lane == src) w += v;
        }
        for (uint32_t o = G >> 1; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
        if (gl == 0 && x < n && !later) finish(x, ne, w);
    }
    __syncthreads();
    const uint32_t nlong = min(s_nlong, kLongRows);
    if (nlong) {
        for (uint32_t i = 0; i < nlong; i++) {
            const uint3 l = s_long[i];
            unsigned long long v = 0;
#pragma unroll 4
            for (uint32_t k = threadIdx.x; k < l.z - l.y; k += blockDim.x) v += candidates(l.y + k);
            v = warp_sum(v);
            if (lane == 0) atomicAdd(&s_w[i], v);
        }
        __syncthreads();
        if (threadIdx.x < nlong) finish(s_long[threadIdx.x].x, s_long[threadIdx.x].z - s_long[threadIdx.x].y, s_w[threadIdx.x]);
        __syncthreads();
    }
    if (threadIdx.x < 6 && s_acc[threadIdx.x]) atomicAdd(threadIdx.x ? &outj_cls[threadIdx.x] : outj, s_acc[threadIdx.x]);
    if (threadIdx.x < kRowBuckets && s_n[threadIdx.x])
        atomicAdd(&nbucket[threadIdx.x], (unsigned long long)s_n[threadIdx.x]);
}
// Lanes a row (log2) for rows of `per_row` entries on average.  Both CSRs and
// the row work of 4M x 500K tuples, us with 4, 8, 16 and 32 lanes: 2 a row 296
// 309 397 606, 5 a row 246 242 272 363, 12 a row 214 211 215 258, 40 a row 192
// 189 187 194, 64 a row 197 190 188 188.
inline uint32_t row_work_lanes(double per_row) { return per_row > 64 ? 5 : (per_row > 24 ? 4 : (per_row > 8 ? 3 : 2)); }

// Every row into its bucket's list: list_w, list_b (buckets 1, 2, 3 in
// turn), list_m (4 then 5: the huge rows first) and list_t.  k_row_work has
// counted the buckets (nbucket), so where each starts is known; a CTA ranks
// its kListTile rows in shared memory and takes one range of each bucket from
// its cursor.  One launch (a prefix sum per bucket was three each).  Rows of
// a tile stay in order and together; the order of tiles is unspecified.  The
// class counts go to n[1..5] and nb[0..2].  Buckets are stored from k0 on
// (many-query passes keep two families of rows in one array).
constexpr uint32_t kListItems = 8, kListTile = 256 * kListItems;
static __global__ void __launch_bounds__(256) k_row_lists(const uint8_t* __restrict__ bucket, uint32_t n, uint32_t k0,
                                                          const unsigned long long* __restrict__ nbucket,
                                                          unsigned long long* cursor, uint32_t* __restrict__ lists,
                                                          unsigned long long* nrows, unsigned long long* nrows_b) {
    __shared__ uint32_t s_n[kRowBuckets + 1];
    __shared__ uint32_t* s_at[kRowBuckets];
    if (threadIdx.x <= kRowBuckets) s_n[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t t0 = (uint64_t)blockIdx.x * kListTile;
    const uint32_t lane = lane_id();
    uint32_t b[kListItems], rank[kListItems];
#pragma unroll
    for (uint32_t k = 0; k < kListItems; k++) {
        const uint64_t x = t0 + k * 256 + threadIdx.x;
        b[k] = x < n ? bucket[x] - k0 : kRowBuckets;
        b[k] = b[k] < kRowBuckets ? b[k] : kRowBuckets;
    }
#pragma unroll
    for (uint32_t k = 0; k < kListItems; k++) {
        const unsigned grp = __match_any_sync(0xffffffffu, b[k]);
        const int leader = __ffs(grp) - 1;
        uint32_t r = 0;
        if ((int)lane == leader) r = atomicAdd(&s_n[b[k]], (uint32_t)__popc(grp));
        rank[k] = __shfl_sync(0xffffffffu, r, leader) + __popc(grp & lanemask_lt());
    }
    __syncthreads();
    if (threadIdx.x < kRowBuckets) {
        const uint32_t q = threadIdx.x;
        uint32_t* list = lists + (q == 0 ? 0ull : (q <= 3 ? 1ull : (q <= 5 ? 2ull : 3ull))) * n;
        unsigned long long at = s_n[q] ? atomicAdd(&cursor[q], (unsigned long long)s_n[q]) : 0ull;
        if (q == 2 || q == 3) at += nbucket[1];
        if (q == 3) at += nbucket[2];
        if (q == 5) at += nbucket[4];
        s_at[q] = list + at;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        nrows[1] = nbucket[0];
        nrows[2] = nbucket[1] + nbucket[2] + nbucket[3];
        nrows[3] = nbucket[5];
        nrows[4] = nbucket[4];
        nrows[5] = nbucket[6];
        for (int k = 0; k < 3; k++) nrows_b[k] = nbucket[1 + k];
    }
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < kListItems; k++)
        if (b[k] < kRowBuckets) s_at[b[k]][rank[k]] = (uint32_t)(t0 + k * 256 + threadIdx.x);
}

// Output offsets from the rows' distinct counts.  A row has up to m pairs, so
// 4096 rows pass 2^32 from 2^20 pairs a row on.
struct RowCountSrc {
    using Sum = uint64_t;
    const uint32_t* a;
    __device__ uint64_t operator()(uint64_t i) const { return a[i]; }
};
struct OffDst {
    unsigned long long* off;
    __device__ void operator()(uint64_t i, uint64_t e, uint64_t) const { off[i] = e; }
};

}  // namespace dim3g
