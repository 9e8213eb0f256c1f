// aggregate.cuh -- COUNT(*) GROUP BY (x, z) (SpmmAggregate with a COUNT
// plug-in, dim3.hpp:1271-1310).
//
// Each row is expanded with a counter per distinct z and then emits every
// (x, z, count).  Counts are exact: each expansion candidate is one joining
// (R tuple, S tuple) pair.  Row forms:
//   tiny rows    packs of rows to a warp (packed.cuh), a shared map row, z ->
//                count, groups staged across packs; without a cursor a warp a
//                row
//   map rows     one CTA a row, a shared map z -> count (or a counter per z
//                where the domain is small), CTA width and map by row size
//   ranked rows  one CTA a row and z tile: a bitmap of the z that occur, their
//                ranks by popcount, then a counter per rank -- two passes over
//                the candidates, memory by the distinct z and not the domain
// The groups go to a reserved range of a global cursor (rows in any order), or,
// for ordered output and callers that size the output first, to the row's
// exact offset from a count pass.
#pragma once
#include "common.cuh"
#include "expand.cuh"
#include "packed.cuh"
#include "single.cuh"

namespace dim3g {

struct AggOut {
    unsigned long long* cnt;  // one count per output pair
    SumAcc sum;               // sum.tiles set: summaries instead of output
    Reserve rs;               // cursor and capacity (cursor null: rows at c.off)
};

// Per-lane sums of a summary.
struct GroupSums {
    unsigned long long g = 0, cs = 0, h = 0;
    __device__ __forceinline__ void add(uint32_t xv, uint32_t zv, uint32_t cnt) {
        g++;
        cs += cnt;
        h += group_hash(xv, zv, cnt);
    }
};

// Shared-memory map slot of z (inserting it if absent).
__device__ __forceinline__ uint32_t smem_map_slot(uint32_t* keys, uint32_t lg, uint32_t z, uint32_t* err) {
    const uint32_t mask = (1u << lg) - 1;
    uint32_t h = (z * 0x9E3779B1u) >> (32 - lg);
    volatile uint32_t* vk = keys;
    for (uint32_t p = 0; p <= mask; p++) {
        uint32_t cur = vk[h];
        if (cur == z) return h;
        if (cur == kEmpty32) {
            uint32_t prev = atomicCAS(&keys[h], kEmpty32, z);
            if (prev == kEmpty32 || prev == z) return h;
        }
        h = (h + 1) & mask;
    }
    raise_error(err, kErrTableFull);
    return 0xFFFFFFFFu;
}

// Counting "sets" for the expansion: they take every candidate and report no
// first insertions (emission happens after the expansion).
struct CountMap {
    uint32_t* keys;
    uint32_t* vals;
    uint32_t lg;
    uint32_t* err;
    __device__ __forceinline__ bool insert(uint32_t z, bool act) {
        if (act) {
            uint32_t s = smem_map_slot(keys, lg, z, err);
            if (s != 0xFFFFFFFFu) atomicAdd(&vals[s], 1u);
        }
        return false;
    }
};
struct CountTile {
    uint32_t* ctr;
    uint32_t lo;
    __device__ __forceinline__ bool insert(uint32_t z, bool act) {
        if (act) atomicAdd(&ctr[z - lo], 1u);
        return false;
    }
};
struct MarkTile {  // ranked rows, first pass
    uint32_t* bm;
    uint32_t lo;
    __device__ __forceinline__ bool insert(uint32_t z, bool act) {
        const uint32_t zl = z - lo;
        if (act) atomicOr(&bm[zl >> 5], 1u << (zl & 31));
        return false;
    }
};
// Ranked rows, second pass: rank of z = set bits below it.  A warp's words
// start at wbase[w >> wsh]; pre[w] counts the bits of the warp's earlier
// words.
struct RankedTile {
    const uint32_t* bm;
    const uint16_t* pre;
    const uint32_t* wbase;
    uint32_t wsh;
    __device__ __forceinline__ uint32_t rank(uint32_t zl) const {
        const uint32_t w = zl >> 5;
        return wbase[w >> wsh] + pre[w] + __popc(bm[w] & ((1u << (zl & 31)) - 1u));
    }
};
struct CountRanked {
    RankedTile t;
    uint32_t lo, r0, n;  // counters of ranks [r0, r0 + n)
    uint32_t* ctr;
    uint32_t* zl;  // the ranks' z: written by the candidate that finds a zero count
    __device__ __forceinline__ bool insert(uint32_t z, bool act) {
        if (act) {
            const uint32_t r = t.rank(z - lo) - r0;
            if (r < n && atomicAdd(&ctr[r], 1u) == 0) zl[r] = z;
        }
        return false;
    }
};
struct CountGlobal {  // ranked rows of many ranks, second pass
    RankedTile t;
    uint32_t lo;
    uint32_t* g;
    __device__ __forceinline__ bool insert(uint32_t z, bool act) {
        if (act) atomicAdd(&g[t.rank(z - lo)], 1u);
        return false;
    }
};
struct NullSink {
    static constexpr bool kValues = false;
    template <uint32_t N>
    __device__ __forceinline__ void take(const uint32_t (&)[N], const uint32_t (&)[N]) {}
    template <uint32_t N>
    __device__ __forceinline__ void take(const uint32_t (&)[N], const uint32_t (&)[N], const uint32_t (&)[N]) {}
};

// A map-class row counts with one counter per z of the whole domain instead
// of a z -> count hash map when the m counters fit the map memory (2^words_lg
// words) and scanning them costs little against the row's candidates
// (m <= 8 u).
__device__ __forceinline__ bool use_row_counters(uint32_t m, uint32_t u, uint32_t words_lg) {
    return (uint64_t)m <= (1ull << words_lg) && (uint64_t)m <= 8ull * u;
}

// Where n groups of row x go (warp-uniform; ~0: nowhere).  Cursor: a
// reservation ending past the capacity writes nothing.  Offsets: the row's
// next n places (*s_pos counts them), checked against its count.
__device__ __forceinline__ unsigned long long group_place(const RowCtx& c, const AggOut& ao, uint32_t x, uint32_t n,
                                                          uint32_t* s_pos) {
    unsigned long long base = 0;
    if (lane_id() == 0) {
        if (ao.rs.cursor) {
            base = atomicAdd(ao.rs.cursor, (unsigned long long)n);
            if (base + n > ao.rs.cap) base = ~0ull;
        } else {
            const uint32_t p = atomicAdd(s_pos, n);
            base = c.off[x] + p;
            if (p + n > c.cnt[x]) {
                raise_error(c.err, kErrOutputBound);
                base = ~0ull;
            }
        }
    }
    return __shfl_sync(0xffffffffu, base, 0);
}

// ------------------------------------------------------------- map rows
// The whole CTA: row x through a map of 2^lg keys and counts at smem.  Called
// after a barrier that follows the previous row; *s_pos is 0 by the first
// barrier in here.
__device__ __forceinline__ void agg_map_row(const RowCtx& c, const AggOut& ao, uint32_t x, uint32_t* smem, uint32_t lg,
                                            CtaChunks* cc, uint32_t* s_pos) {
    const uint32_t nw = blockDim.x >> 5, wib = threadIdx.x >> 5, lane = lane_id();
    const uint32_t u = c.ucap[x], e0 = c.JR_R[x], e1 = c.JR_R[x + 1], ne = e1 - e0;
    const bool direct = use_row_counters(c.m, u, lg + 1);
    uint32_t rl = ceil_log2(2 * u);
    rl = rl < 5 ? 5 : (rl > lg ? lg : rl);
    uint32_t* keys = smem;
    uint32_t* vals = direct ? smem : smem + (1u << rl);
    const uint32_t span = direct ? c.m : 1u << rl;
    uint4* t4 = reinterpret_cast<uint4*>(smem);
    if (direct) {
        for (uint32_t s = threadIdx.x; s < (span + 3) / 4; s += blockDim.x) t4[s] = make_uint4(0, 0, 0, 0);
    } else {
        for (uint32_t s = threadIdx.x; s < span / 4; s += blockDim.x) {
            t4[s] = make_uint4(kEmpty32, kEmpty32, kEmpty32, kEmpty32);
            t4[s + span / 4] = make_uint4(0, 0, 0, 0);
        }
    }
    if (threadIdx.x == 0) *s_pos = 0;
    const uint64_t pol = l2_keep_policy();
    const bool staged = ne <= kRowBlk;
    if (staged) balanced_stage(c, e0, ne, 0, c.T, cc, pol, wib, nw);
    __syncthreads();
    NullSink sink;
    CountTile ct{smem, 0};
    CountMap cm{keys, vals, rl, c.err};
    if (staged) {
        if (direct) balanced_expand(c, ne, ct, sink, cc->st.seg.s0, cc->st.seg.incl, cc->ctot, pol, wib, nw);
        else balanced_expand(c, ne, cm, sink, cc->st.seg.s0, cc->st.seg.incl, cc->ctot, pol, wib, nw);
    } else {
        if (direct) cta_expand_balanced(c, e0, e1, 0, c.T, ct, sink, cc);
        else cta_expand_balanced(c, e0, e1, 0, c.T, cm, sink, cc);
    }
    __syncthreads();
    // the warps' equal parts of the map, whole groups of 32 slots
    const uint32_t per = (((span + nw - 1) / nw) + 31) & ~31u;
    const uint32_t s0 = min(span, wib * per), s1 = min(span, s0 + per);
    const uint32_t xv = c.id2x[x];
    if (ao.sum.tiles) {
        GroupSums gs;
        for (uint32_t s = s0 + lane; s < s1; s += 32) {
            const uint32_t v = vals[s];
            if (v) gs.add(xv, __ldg(&c.id2z[direct ? s : keys[s]]), v);
        }
        ao.sum.commit(xv, gs.g, gs.cs, gs.h);
        return;
    }
    uint32_t n = 0;
    for (uint32_t s = s0 + lane; s < s1; s += 32) n += vals[s] != 0;
    n = __reduce_add_sync(0xffffffffu, n);
    if (n == 0) return;
    unsigned long long base = group_place(c, ao, x, n, s_pos);
    if (base == ~0ull) return;
    for (uint32_t sb = s0; sb < s1; sb += 128) {  // four id gathers in flight
        uint32_t v[4], z[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) {
            const uint32_t s = sb + k * 32 + lane;
            v[k] = s < s1 ? vals[s] : 0u;
            z[k] = v[k] ? __ldg(&c.id2z[direct ? s : keys[s]]) : 0u;
        }
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) {
            const uint32_t b = __ballot_sync(0xffffffffu, v[k] != 0);
            if (v[k]) {
                const unsigned long long pos = base + __popc(b & lanemask_lt());
                st_stream(&c.out[pos], make_uint2(xv, z[k]));
                __stcs(&ao.cnt[pos], (unsigned long long)v[k]);
            }
            base += __popc(b);
        }
    }
}

// ---------------------------------------------------------- ranked rows
// Shared memory of a ranked row: the tile's bitmap words (padded to the
// warps' word ranges), a 16-bit prefix a word, then as many (counter, z)
// pairs as fit.
struct RankLayout {
    uint32_t wsh;    // words a warp ranks (log2, at least 7)
    uint32_t words;  // bitmap words, a multiple of the warps' ranges
    uint32_t cap;    // ranks counted at a time
};
__host__ __device__ inline RankLayout rank_layout(uint32_t tile_width, uint32_t warps, size_t smem) {
    RankLayout l;
    const uint32_t w = (tile_width + 31) / 32, per = (w + warps - 1) / warps;
    l.wsh = 7;
    while ((1u << l.wsh) < per) l.wsh++;
    l.words = ((w + (1u << l.wsh) - 1) >> l.wsh) << l.wsh;
    l.cap = (uint32_t)((smem - (size_t)l.words * 6) / 8);
    return l;
}

// A row (or row and tile) of the ranked class: item number, row, its entries
// and first value, tile.
struct RankHead {
    uint64_t item;
    uint32_t x, e0, e1, xv, t;
};
__device__ __forceinline__ RankHead rank_head(const RowCtx& c, uint64_t item, uint32_t x, uint32_t t) {
    return RankHead{item, x, c.JR_R[x], c.JR_R[x + 1], c.id2x[x], t};
}

// The whole CTA: row h.x over tile t.  Groups go to the cursor, or (offsets)
// to the row's next places.  Called after a barrier that follows the previous
// row; *s_pos as the caller keeps it for the row.  ahead() runs on thread 0
// during the first pass (the other warps take its share of the pieces).
// g: the CTA's tile_width counters in global memory, all zero between calls,
// or null.  A tile of more than two windows of ranks counts there in one walk
// instead of one walk a window.  (A query pass of 600 rows, windows of 23K
// ranks, there and in windows: 28K distinct z a row 0.62 and 0.48 ms, 40K 0.77
// and 0.64, 52K 0.95 and 1.01, 90K 1.54 and 2.04.)
template <class Ahead>
__device__ __forceinline__ void agg_ranked_tile(const RowCtx& c, const AggOut& ao, const RankHead& h, uint32_t t,
                                                uint32_t* smem, const RankLayout& l, CtaChunks* cc, uint32_t* s_pos,
                                                uint32_t* s_wbase, unsigned long long* s_base, uint32_t* g,
                                                Ahead ahead) {
    const uint32_t nw = blockDim.x >> 5, wib = threadIdx.x >> 5, lane = lane_id();
    const uint32_t x = h.x, e0 = h.e0, e1 = h.e1, ne = e1 - e0, lo = t * c.tile_width, xv = h.xv;
    uint32_t* bm = smem;
    uint16_t* pre = reinterpret_cast<uint16_t*>(smem + l.words);
    uint32_t* ctr = smem + l.words + l.words / 2;
    uint32_t* zl = ctr + l.cap;
    const uint64_t pol = l2_keep_policy();
    const bool staged = ne <= kRowBlk;
    NullSink sink;
    uint4* b4 = reinterpret_cast<uint4*>(bm);
    for (uint32_t w = threadIdx.x; w < l.words / 4; w += blockDim.x) b4[w] = make_uint4(0, 0, 0, 0);
    if (staged) balanced_stage(c, e0, ne, t, t + 1, cc, pol, wib, nw);
    if (threadIdx.x == 0) cc->n = 0;
    __syncthreads();
    if (threadIdx.x == 0) ahead();
    __syncwarp();
    MarkTile mark{bm, lo};
    if (staged) balanced_expand(c, ne, mark, sink, cc->st.seg.s0, cc->st.seg.incl, cc->ctot, pol, wib, nw, &cc->n, kDynPiece);
    else cta_expand_balanced(c, e0, e1, t, t + 1, mark, sink, cc);
    __syncthreads();
    // ranks: every warp's words, then the warps' bases
    const uint32_t w0 = wib << l.wsh, w1 = min(l.words, w0 + (1u << l.wsh));
    uint32_t run = 0;
    for (uint32_t w = w0 + 4 * lane; w < w1; w += 128) {  // four words a lane
        const uint4 b = b4[w >> 2];
        const uint32_t n0 = __popc(b.x), n1 = n0 + __popc(b.y), n2 = n1 + __popc(b.z), n3 = n2 + __popc(b.w);
        const uint32_t inc = warp_incl_scan(n3), p = run + inc - n3;
        *reinterpret_cast<uint2*>(pre + w) = make_uint2(p | (p + n0) << 16, (p + n1) | (p + n2) << 16);
        run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) s_wbase[wib] = run;
    if (threadIdx.x == 0) cc->n = 0;
    __syncthreads();
    if (wib == 0) {
        const uint32_t v = lane < nw ? s_wbase[lane] : 0u, inc = warp_incl_scan(v);
        const uint32_t d = __shfl_sync(0xffffffffu, inc, 31);
        __syncwarp();
        s_wbase[lane] = inc - v;
        if (lane == 0) s_wbase[32] = d;
    }
    __syncthreads();
    const uint32_t d = s_wbase[32];
    // the reservation's round trip passes while the other warps set up the
    // window; read after the next barriers
    if (wib == 0 && d && !ao.sum.tiles) {
        const unsigned long long base = group_place(c, ao, x, d, s_pos);
        if (lane == 0) *s_base = base;
    }
    GroupSums gs;
    const RankedTile rt{bm, pre, s_wbase, l.wsh};
    if (g && d > 2 * l.cap) {
        __syncthreads();  // *s_base; cc->n
        CountGlobal cg{rt, lo, g};
        if (staged) balanced_expand(c, ne, cg, sink, cc->st.seg.s0, cc->st.seg.incl, cc->ctot, pol, wib, nw, &cc->n, kDynPiece);
        else cta_expand_balanced(c, e0, e1, t, t + 1, cg, sink, cc);
        __syncthreads();
        const unsigned long long base = ao.sum.tiles ? 0ull : *s_base;
        for (uint32_t wb = w0; wb < w1; wb += 4) {  // a warp's own words, a lane a bit
            uint32_t r[4], v[4], z[4];
            bool on[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) {
                const uint32_t b = bm[wb + k];
                on[k] = b >> lane & 1u;
                r[k] = s_wbase[wib] + pre[wb + k] + __popc(b & lanemask_lt());
                v[k] = on[k] ? __ldcg(&g[r[k]]) : 0u;
                z[k] = on[k] ? __ldg(&c.id2z[lo + (wb + k) * 32 + lane]) : 0u;
            }
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) {
                if (!on[k]) continue;
                __stcg(&g[r[k]], 0u);
                if (ao.sum.tiles) {
                    gs.add(xv, z[k], v[k]);
                } else if (base != ~0ull) {
                    st_stream(&c.out[base + r[k]], make_uint2(xv, z[k]));
                    __stcs(&ao.cnt[base + r[k]], (unsigned long long)v[k]);
                }
            }
        }
        if (threadIdx.x == 0) cc->n = 0;
        __syncthreads();  // the next row's bitmap
        if (ao.sum.tiles) ao.sum.commit(xv, gs.g, gs.cs, gs.h);
        return;
    }
    for (uint32_t r0 = 0; r0 < d; r0 += l.cap) {
        const uint32_t n = min(l.cap, d - r0);
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) ctr[i] = 0;
        __syncthreads();
        CountRanked cr{rt, lo, r0, n, ctr, zl};
        if (staged) balanced_expand(c, ne, cr, sink, cc->st.seg.s0, cc->st.seg.incl, cc->ctot, pol, wib, nw, &cc->n, kDynPiece);
        else cta_expand_balanced(c, e0, e1, t, t + 1, cr, sink, cc);
        __syncthreads();
        if (ao.sum.tiles) {
            for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) gs.add(xv, __ldg(&c.id2z[zl[i]]), ctr[i]);
        } else if (*s_base != ~0ull) {
            const unsigned long long base = *s_base + r0;
            for (uint32_t ib = threadIdx.x; ib < n; ib += 4 * blockDim.x) {  // four id gathers in flight
                uint32_t z[4], v[4];
#pragma unroll
                for (uint32_t k = 0; k < 4; k++) {
                    const uint32_t i = ib + k * blockDim.x;
                    z[k] = i < n ? __ldg(&c.id2z[zl[i]]) : 0u;
                    v[k] = i < n ? ctr[i] : 0u;
                }
#pragma unroll
                for (uint32_t k = 0; k < 4; k++) {
                    const uint32_t i = ib + k * blockDim.x;
                    if (i < n) {
                        st_stream(&c.out[base + i], make_uint2(xv, z[k]));
                        __stcs(&ao.cnt[base + i], (unsigned long long)v[k]);
                    }
                }
            }
        }
        if (threadIdx.x == 0) cc->n = 0;
        __syncthreads();  // the next window's counters; the next row's bitmap
    }
    if (ao.sum.tiles) ao.sum.commit(xv, gs.g, gs.cs, gs.h);
}

// ---------------------------------------------------------- direct rows
// Rows of many candidates: a counter per z of a tile of at most
// 2^kAggDirectLg ids, so the candidates are walked once -- ranked rows walk
// them twice and once more for every window of ranks past the first, which is
// what a dense row pays for most (a 1/16 slice of the 16M-tuple COUNT on the
// sparse kernels, 830K candidates a row over 1M z: ranked 47 s, direct 0.65).
constexpr uint32_t kAggDirectLg = 15;
// The whole CTA, as agg_ranked_tile; ctr holds a word a z of the tile.  The
// caller commits a summary's sums, once a row.
template <class Ahead>
__device__ __forceinline__ void agg_direct_tile(const RowCtx& c, const AggOut& ao, const RankHead& h, uint32_t t,
                                                uint32_t* ctr, CtaChunks* cc, uint32_t* s_pos, uint32_t* s_wbase,
                                                unsigned long long* s_base, GroupSums& gs, Ahead ahead) {
    const uint32_t nw = blockDim.x >> 5, wib = threadIdx.x >> 5, lane = lane_id();
    const uint32_t ne = h.e1 - h.e0, lo = t * c.tile_width, width = min(c.tile_width, c.m - lo), xv = h.xv;
    const uint64_t pol = l2_keep_policy();
    const bool staged = ne <= kRowBlk;
    NullSink sink;
    for (uint32_t i = threadIdx.x; i < width; i += blockDim.x) ctr[i] = 0;
    if (staged) balanced_stage(c, h.e0, ne, t, t + 1, cc, pol, wib, nw);
    if (threadIdx.x == 0) cc->n = 0;
    __syncthreads();
    if (threadIdx.x == 0) ahead();
    __syncwarp();
    CountTile set{ctr, lo};
    if (staged) balanced_expand(c, ne, set, sink, cc->st.seg.s0, cc->st.seg.incl, cc->ctot, pol, wib, nw, &cc->n, 0);
    else cta_expand_balanced(c, h.e0, h.e1, t, t + 1, set, sink, cc);
    __syncthreads();
    const uint32_t per = (((width + nw - 1) / nw) + 31) & ~31u, s0 = min(width, wib * per), s1 = min(width, s0 + per);
    if (ao.sum.tiles) {
        for (uint32_t i = s0 + lane; i < s1; i += 32)
            if (ctr[i]) gs.add(xv, __ldg(&c.id2z[lo + i]), ctr[i]);
        __syncthreads();  // the next tile's counters
        return;
    }
    // the warps' places in one reservation a tile
    uint32_t n = 0;
    for (uint32_t i = s0 + lane; i < s1; i += 32) n += ctr[i] != 0;
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0) s_wbase[wib] = n;
    __syncthreads();
    if (wib == 0) {
        const uint32_t v = lane < nw ? s_wbase[lane] : 0u, inc = warp_incl_scan(v);
        const uint32_t d = __shfl_sync(0xffffffffu, inc, 31);
        __syncwarp();
        s_wbase[lane] = inc - v;
        const unsigned long long base = d ? group_place(c, ao, h.x, d, s_pos) : ~0ull;
        if (lane == 0) *s_base = base;
    }
    __syncthreads();
    if (*s_base != ~0ull) {
        unsigned long long base = *s_base + s_wbase[wib];
        for (uint32_t sb = s0; sb < s1; sb += 128) {  // four id gathers in flight
            uint32_t v[4], z[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) {
                const uint32_t i = sb + k * 32 + lane;
                v[k] = i < s1 ? ctr[i] : 0u;
                z[k] = v[k] ? __ldg(&c.id2z[lo + i]) : 0u;
            }
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) {
                const uint32_t b = __ballot_sync(0xffffffffu, v[k] != 0);
                if (v[k]) {
                    const unsigned long long pos = base + __popc(b & lanemask_lt());
                    st_stream(&c.out[pos], make_uint2(xv, z[k]));
                    __stcs(&ao.cnt[pos], (unsigned long long)v[k]);
                }
                base += __popc(b);
            }
        }
    }
    __syncthreads();  // the next tile's counters
}

// ------------------------------------------------------------ tiny rows
// (x, z, count) groups staged across the rows of one warp and one query,
// reserved once per `cap` groups (see PairStageSink).
struct GroupStage {
    uint2* pairs;      // cap (x value, z value)
    uint32_t* counts;  // cap counts
    uint2* out;
    unsigned long long* out_cnt;
    Reserve rs;
    uint32_t cap;      // at least 32
    uint32_t n = 0;
    __device__ __forceinline__ void flush() {
        if (n == 0) return;
        unsigned long long base = 0;
        if (lane_id() == 0) base = atomicAdd(rs.cursor, (unsigned long long)n);
        base = __shfl_sync(0xffffffffu, base, 0);
        __syncwarp();
        if (base + n <= rs.cap)
            for (uint32_t i = lane_id(); i < n; i += 32) {
                st_stream(&out[base + i], pairs[i]);
                __stcs(&out_cnt[base + i], (unsigned long long)counts[i]);
            }
        __syncwarp();
        n = 0;
    }
    // warp-collective: the lanes with `have` add one group each
    __device__ __forceinline__ void add(bool have, uint32_t xv, uint32_t zv, uint32_t cnt) {
        const uint32_t b = __ballot_sync(0xffffffffu, have);
        if (!b) return;
        if (n + __popc(b) > cap) flush();
        if (have) {
            const uint32_t pos = n + __popc(b & lanemask_lt());
            pairs[pos] = make_uint2(xv, zv);
            counts[pos] = cnt;
        }
        n += __popc(b);
        __syncwarp();
    }
};

// Slots (log2) of a warp's map, staged groups, shared words a warp.
constexpr uint32_t kAggPackLg = 9, kAggPackStage = 128;
constexpr size_t kAggPackWords = ((size_t)2 << kAggPackLg) + 3 * kAggPackStage;
static_assert(kTinyU <= (1u << (kAggPackLg - 1)), "a small row fits a pack");

// Rows of lanes [lo, hi) (x: the lane's row) as packs into the warp's map.
__device__ __forceinline__ void agg_pack_rows(const RowCtx& c, uint32_t x, uint32_t lo, uint32_t hi, uint32_t* keys,
                                              GroupStage& gs) {
    const uint32_t lane = lane_id();
    uint32_t u = 0, e0 = 0, ne = 0, xv = 0;
    if (lane >= lo && lane < hi) {
        u = c.ucap[x];
        e0 = c.JR_R[x];
        ne = c.JR_R[x + 1] - e0;
        xv = c.id2x[x];
    }
    for (uint32_t first = lo; first < hi;) {
        uint32_t sum;
        const uint32_t end = pack_end(u, first, hi, c.m, 1u << (kAggPackLg - 1), &sum);
        const bool in = lane >= first && lane < end;
        uint32_t lg = ceil_log2(2 * sum);
        lg = lg < 5 ? 5 : lg;
        // a counter a row and z where those are no more than the map's words
        const uint64_t cells = (uint64_t)(end - first) * c.m;
        const bool direct = cells <= (2u << lg);
        const uint32_t span = direct ? (uint32_t)cells : 1u << lg;
        uint32_t* vals = direct ? keys : keys + (1u << lg);
        for (uint32_t s = lane; s < span; s += 32) {
            keys[s] = direct ? 0u : kEmpty32;
            if (!direct) vals[s] = 0;
        }
        __syncwarp();
        NullSink sink;
        const uint32_t n = in ? ne : 0u, key0 = in ? (lane - first) * c.m : 0u;
        if (direct) {
            CountTile set{keys, 0};
            pack_expand<false>(c, e0, n, key0, xv, set, sink);
        } else {
            CountMap set{keys, vals, lg, c.err};
            pack_expand<false>(c, e0, n, key0, xv, set, sink);
        }
        __syncwarp();
        for (uint32_t sb = 0; sb < span; sb += 32) {
            const uint32_t s = sb + lane, v = s < span ? vals[s] : 0u;
            const bool have = v != 0;
            const uint32_t key = have ? (direct ? s : keys[s]) : 0u, r = have ? key / c.m : 0u;
            const uint32_t gx = __shfl_sync(0xffffffffu, xv, first + r);
            gs.add(have, gx, have ? __ldg(&c.id2z[key - r * c.m]) : 0u, v);
        }
        __syncwarp();
        first = end;
    }
}

// ------------------------------------------------------------- one join
static __global__ void __launch_bounds__(256, 4) k_agg_pack(RowCtx c, AggOut ao, const uint32_t* __restrict__ rows,
                                                         const unsigned long long* __restrict__ nrows_p) {
    extern __shared__ uint32_t smem[];
    const uint32_t nw = blockDim.x >> 5, wib = threadIdx.x >> 5, lane = lane_id();
    uint32_t* keys = smem + (size_t)wib * kAggPackWords;
    uint32_t* stage = keys + (2u << kAggPackLg);
    GroupStage gs{reinterpret_cast<uint2*>(stage), stage + 2 * kAggPackStage, c.out, ao.cnt, ao.rs, kAggPackStage};
    const uint32_t nrows = (uint32_t)*nrows_p, warps = gridDim.x * nw;
    uint32_t take = (nrows + warps - 1) / warps;
    take = take > 32 ? 32 : take;
    for (uint64_t r0 = (uint64_t)(blockIdx.x * nw + wib) * take; r0 < nrows; r0 += (uint64_t)warps * take) {
        const uint32_t n = (uint32_t)min((uint64_t)take, nrows - r0);
        agg_pack_rows(c, lane < n ? rows[r0 + lane] : 0u, 0, n, keys, gs);
    }
    gs.flush();
}

// Tiny rows without a cursor -- at exact offsets, or hashed into a summary,
// whose sums are committed once a row -- one warp a row, with a counter per z
// or a map of its own.  (2.9M tuples in 720K rows of about 20 candidates, a
// summary, whole call: 4.3 ms with a CTA for each row, 2.2 so.)
static __global__ void __launch_bounds__(256) k_agg_warp(RowCtx c, AggOut ao, const uint32_t* __restrict__ rows,
                                                         const unsigned long long* __restrict__ nrows_p) {
    extern __shared__ uint32_t smem[];
    const uint32_t nw = blockDim.x >> 5, wib = threadIdx.x >> 5, lane = lane_id();
    uint32_t* keys = smem + ((size_t)wib << (kAggPackLg + 1));
    const uint32_t nrows = (uint32_t)*nrows_p;
    NullSink sink;
    for (uint32_t ri = blockIdx.x * nw + wib; ri < nrows; ri += gridDim.x * nw) {
        const uint32_t x = rows[ri], u = c.ucap[x], xv = c.id2x[x];
        const bool direct = use_row_counters(c.m, u, kAggPackLg + 1);
        uint32_t rl = ceil_log2(2 * u);
        rl = rl < 5 ? 5 : rl;
        const uint32_t span = direct ? c.m : 1u << rl;
        uint32_t* vals = direct ? keys : keys + span;
        for (uint32_t s = lane; s < span; s += 32) {
            keys[s] = direct ? 0u : kEmpty32;
            if (!direct) vals[s] = 0;
        }
        __syncwarp();
        if (direct) {
            CountTile set{keys, 0};
            warp_expand(c, c.JR_R[x], c.JR_R[x + 1], 0, 0, 0, c.T, set, sink);
        } else {
            CountMap set{keys, vals, rl, c.err};
            warp_expand(c, c.JR_R[x], c.JR_R[x + 1], 0, 0, 0, c.T, set, sink);
        }
        __syncwarp();
        if (ao.sum.tiles) {
            GroupSums gs;
            for (uint32_t s = lane; s < span; s += 32) {
                const uint32_t v = vals[s];
                if (v) gs.add(xv, __ldg(&c.id2z[direct ? s : keys[s]]), v);
            }
            ao.sum.commit(xv, gs.g, gs.cs, gs.h);
        } else {
            const unsigned long long base = c.off[x];
            const uint32_t lim = c.cnt[x];
            uint32_t pos = 0;
            for (uint32_t sb = 0; sb < span; sb += 32) {
                const uint32_t s = sb + lane, v = s < span ? vals[s] : 0u, b = __ballot_sync(0xffffffffu, v != 0);
                if (v) {
                    const uint32_t p = pos + __popc(b & lanemask_lt());
                    if (p < lim) {
                        st_stream(&c.out[base + p], make_uint2(xv, __ldg(&c.id2z[direct ? s : keys[s]])));
                        __stcs(&ao.cnt[base + p], (unsigned long long)v);
                    } else {
                        raise_error(c.err, kErrOutputBound);
                    }
                }
                pos += __popc(b);
            }
        }
        __syncwarp();
    }
}

// Map rows rows[skip0 + skip1 + i], i < *nrows_p (skips: device counts, either
// may be null), maps of up to 2^lg keys; row counter c.next_row[ctr].
static __global__ void __launch_bounds__(1024, 1) k_agg_map(RowCtx c, AggOut ao, const uint32_t* __restrict__ rows,
                                                         const unsigned long long* __restrict__ nrows_p, uint32_t lg,
                                                         const unsigned long long* skip0,
                                                         const unsigned long long* skip1, uint32_t ctr) {
    extern __shared__ uint32_t smem[];
    __shared__ uint32_t s_pos, s_row;
    __shared__ CtaChunks s_cc;
    const uint32_t nrows = (uint32_t)*nrows_p;
    rows += (skip0 ? *skip0 : 0ull) + (skip1 ? *skip1 : 0ull);
    for (uint32_t ri = cta_next_row(&c.next_row[ctr], &s_row); ri < nrows; ri = cta_next_row(&c.next_row[ctr], &s_row))
        agg_map_row(c, ao, rows[ri], smem, lg, &s_cc, &s_pos);
}

// Ranked rows (classes 4, then 3).  Cursor and summaries: one CTA a row and
// tile, so a huge row's tiles run side by side; offsets, and the summaries of
// direct rows (their sums meet in a few addresses, once a row): one CTA a row.  The
// next item is claimed and its header loaded during the current one.
// FORM: direct rows (`l` and `ctr` unused), ranked rows in windows (ctr
// unused), or ranked rows with every CTA's counters for agg_ranked_tile at
// ctr.  (Without a use for them they cost registers: count_1m 3.41 and 3.48
// ms.)
enum RankForm { kRankDirect, kRankWindows, kRankCounters };
template <RankForm FORM>
static __global__ void __launch_bounds__(1024, 1) k_agg_ranked(RowCtx c, AggOut ao, const uint32_t* __restrict__ rows,
                                                            const unsigned long long* __restrict__ n3,
                                                            const unsigned long long* __restrict__ n4, RankLayout l,
                                                            unsigned long long* next_item, uint32_t* ctr) {
    extern __shared__ uint32_t smem[];
    __shared__ uint32_t s_pos, s_wbase[33];
    __shared__ unsigned long long s_base;
    __shared__ RankHead s_head[2];
    __shared__ CtaChunks s_cc;
    const uint32_t per = ao.rs.cursor || (ao.sum.tiles && FORM != kRankDirect) ? c.T : 1u;
    const TileItems it{*n3 + *n4, per};
    auto claim = [&](RankHead* dst) {
        const uint64_t i = atomicAdd(next_item, 1ull);
        *dst = i < it.count() ? rank_head(c, i, rows[it.row(i)], it.tile(i)) : RankHead{i, 0, 0, 0, 0, 0};
    };
    if (threadIdx.x == 0) claim(&s_head[0]);
    __syncthreads();
    for (uint32_t k = 0;; k ^= 1) {
        const RankHead h = s_head[k];
        if (h.item >= it.count()) break;
        if (threadIdx.x == 0) s_pos = 0;
        const uint32_t t0 = h.t, t1 = per == c.T ? t0 + 1 : c.T;
        GroupSums gs;
        for (uint32_t t = t0; t < t1; t++) {
            auto ahead = [&] {
                if (t == t0) claim(&s_head[k ^ 1]);
            };
            if (FORM == kRankDirect) agg_direct_tile(c, ao, h, t, smem, &s_cc, &s_pos, s_wbase, &s_base, gs, ahead);
            else agg_ranked_tile(c, ao, h, t, smem, l, &s_cc, &s_pos, s_wbase, &s_base,
                                 FORM == kRankCounters ? ctr + (size_t)blockIdx.x * c.tile_width : nullptr, ahead);
            __syncthreads();
        }
        if (FORM == kRankDirect && ao.sum.tiles) ao.sum.commit(h.xv, gs.g, gs.cs, gs.h);
        __syncthreads();
    }
}

}  // namespace dim3g
