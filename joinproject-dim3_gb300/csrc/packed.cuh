// packed.cuh -- small rows, many to a warp.
//
// A row with a few entries and a few dozen candidates leaves most lanes of a
// warp idle, and its chain of dependent loads (row, entries, S bounds,
// candidates) is the time.  Here a warp takes rows of its list 32 at a time,
// one header a lane, and expands as many consecutive ones together as one
// table holds (a pack): the pack's entries are flattened over the lanes, then
// their candidates.  The table's key is row * m + z, row the row's place in
// the pack (a pack takes at most (2^32 - 1) / m rows), so one table keeps the
// rows apart.
//
// 1M rows of 10 entries and 100 candidates: 1185 us with a warp a row (two
// launches, tables of 2^8 and 2^11 slots).
#pragma once
#include "common.cuh"
#include "expand.cuh"
#include "single.cuh"

namespace dim3g {

// Slots (log2) of a warp's table, three times the distinct bound of a pack (a
// probe loop runs as long as its longest lane: 1M rows of 100 candidates 930
// us at twice, 865 at three times, 877 at four times and smaller packs); pairs
// a warp stages.  6 KB a warp, so the registers bound the warps in flight.
constexpr uint32_t kPackLg = 10, kPackCap = 340, kPackStage = 256;
static_assert(kTinyU <= kPackCap, "a small row fits a pack");
constexpr size_t kPackWords = ((size_t)1 << kPackLg) + 2 * kPackStage;  // shared words a warp

// Rows of the warp's 32 that can go into one pack, from lane `first` on:
// lanes [first, result).  u: the lane's distinct bound (0 past the end), m:
// the z domain.
__device__ __forceinline__ uint32_t pack_end(uint32_t u, uint32_t first, uint32_t n, uint32_t m, uint32_t cap,
                                             uint32_t* sum) {
    const uint32_t lane = lane_id();
    const uint32_t most = m <= 0xFFFFFFFFu / 32 ? 32u : 0xFFFFFFFFu / m;
    const uint32_t inc = warp_incl_scan(lane >= first && lane < n ? u : 0u);
    const uint32_t fits = __ballot_sync(0xffffffffu, lane >= first && lane < n && inc <= cap && lane - first < most);
    const uint32_t end = 32 - __clz(fits);  // inc is nondecreasing: the fitting lanes are [first, end)
    *sum = __shfl_sync(0xffffffffu, inc, end - 1);
    return end;
}

// Candidates of the pack: the lane's row has entries [e0, e0 + ne) (ne 0:
// none), keys from key0 on and tag xv.
//   set.insert(key, active) -> bool; sink.take(b[], xv[], v[])
template <bool kPair, class Set, class Sink>
__device__ __forceinline__ void pack_expand(const RowCtx& c, uint32_t e0, uint32_t ne, uint32_t key0, uint32_t xv,
                                            Set& set, Sink& sink) {
    const uint64_t pol = l2_keep_policy();
    const uint32_t lane = lane_id();
    const uint32_t inc_e = warp_incl_scan(ne), exc_e = inc_e - ne;
    const uint32_t E = __shfl_sync(0xffffffffu, inc_e, 31);
    for (uint32_t eb = 0; eb < E; eb += 32) {
        const uint32_t ei = min(eb + lane, E - 1);
        uint32_t r = 0;  // the row holding entry ei
#pragma unroll
        for (uint32_t step = 16; step >= 1; step >>= 1)
            if (__shfl_sync(0xffffffffu, inc_e, r + step - 1) <= ei) r += step;
        const uint32_t e = __shfl_sync(0xffffffffu, e0, r) + (ei - __shfl_sync(0xffffffffu, exc_e, r));
        const uint32_t ek = __shfl_sync(0xffffffffu, key0, r), ex = __shfl_sync(0xffffffffu, xv, r);
        uint32_t s0 = 0, len = 0;
        if (eb + lane < E) {
            const uint64_t row = (uint64_t)ld_keep(&c.IC_R[e], pol) * c.T;
            s0 = ld_keep(&c.JR_S[row], pol);
            len = ld_keep(&c.JR_S[row + c.T], pol) - s0;
        }
        const uint32_t inc = warp_incl_scan(len), exc = inc - len;
        const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
        // long segments: the lanes stride each, without a search a candidate
        uint32_t segs = __ballot_sync(0xffffffffu, len != 0);
        if (total >= kFlatAvgMax * __popc(segs)) {
            for (; segs; segs &= segs - 1) {
                const int k = __ffs(segs) - 1;
                const uint32_t ks0 = __shfl_sync(0xffffffffu, s0, k), klen = __shfl_sync(0xffffffffu, len, k);
                const uint32_t kk = __shfl_sync(0xffffffffu, ek, k), kx = __shfl_sync(0xffffffffu, ex, k);
                for (uint32_t jb = 0; jb < klen; jb += 32 * kUnroll) {
                    uint32_t z[kUnroll], v[kUnroll], x[kUnroll], b[kUnroll];
#pragma unroll
                    for (uint32_t u = 0; u < kUnroll; u++) {
                        const uint32_t j = jb + u * 32 + lane;
                        x[u] = kx;
                        load_cand<kPair, Sink::kValues>(c, ks0 + j, j < klen, pol, z[u], v[u]);
                    }
#pragma unroll
                    for (uint32_t u = 0; u < kUnroll; u++)
                        b[u] = jb + u * 32 < klen ? __ballot_sync(0xffffffffu, set.insert(kk + z[u], z[u] != kEmpty32)) : 0u;
                    sink.take(b, x, v);
                }
            }
            continue;
        }
        for (uint32_t cb = 0; cb < total; cb += 32 * kUnroll) {
            uint32_t z[kUnroll], v[kUnroll], key[kUnroll], x[kUnroll], b[kUnroll];
#pragma unroll
            for (uint32_t u = 0; u < kUnroll; u++) {
                const uint32_t cc = cb + u * 32 + lane;
                const bool act = cc < total;
                const uint32_t ci = act ? cc : cb;
                uint32_t k = 0;
#pragma unroll
                for (uint32_t step = 16; step >= 1; step >>= 1)
                    if (__shfl_sync(0xffffffffu, inc, k + step - 1) <= ci) k += step;
                const uint32_t j = __shfl_sync(0xffffffffu, s0, k) + (ci - __shfl_sync(0xffffffffu, exc, k));
                key[u] = __shfl_sync(0xffffffffu, ek, k);
                x[u] = __shfl_sync(0xffffffffu, ex, k);
                load_cand<kPair, Sink::kValues>(c, j, act, pol, z[u], v[u]);
            }
#pragma unroll
            for (uint32_t u = 0; u < kUnroll; u++)
                b[u] = cb + u * 32 < total
                           ? __ballot_sync(0xffffffffu, set.insert(key[u] + z[u], z[u] != kEmpty32))
                           : 0u;
            sink.take(b, x, v);
        }
    }
}

// The rows of lanes [lo, hi) (x: the lane's row) as packs through the warp's
// table into the sink.  sink.tag(c, x): what the sink is given with each of
// the row's candidates.
template <class Sink>
__device__ __forceinline__ void pack_rows(const RowCtx& c, uint32_t x, uint32_t lo, uint32_t hi, uint32_t* tab,
                                          Sink& sink) {
    const uint32_t lane = lane_id();
    uint32_t u = 0, e0 = 0, ne = 0, tag = 0;
    if (lane >= lo && lane < hi) {
        u = c.ucap[x];
        e0 = c.JR_R[x];
        ne = c.JR_R[x + 1] - e0;
        tag = sink.tag(c, x);
    }
    for (uint32_t first = lo; first < hi;) {
        uint32_t sum;
        const uint32_t end = pack_end(u, first, hi, c.m, kPackCap, &sum);
        const bool in = lane >= first && lane < end;
        const uint32_t key0 = in ? (lane - first) * c.m : 0u, n = in ? ne : 0u;
        const uint32_t rows = end - first;
        uint32_t lg = ceil_log2(3 * sum);
        lg = lg < 5 ? 5 : lg;
        // a bitmap over the pack's rows x z domain where it is no larger
        const uint64_t bits = (uint64_t)rows * c.m;
        const bool bm = bits <= (32ull << lg);
        const uint32_t nclr = bm ? row_bitmap_words((uint32_t)bits) : 1u << lg;
        const uint32_t fill = bm ? 0u : kEmpty32;
        uint4* t4 = reinterpret_cast<uint4*>(tab);
        for (uint32_t s = lane; s < nclr / 4; s += 32) t4[s] = make_uint4(fill, fill, fill, fill);
        __syncwarp();
        if (bm) {
            TileBitmap set{tab, 0};
            if (Sink::kValues && c.ISV) pack_expand<true>(c, e0, n, key0, tag, set, sink);
            else pack_expand<false>(c, e0, n, key0, tag, set, sink);
        } else {
            HashSet set{tab, lg, c.err};
            if (Sink::kValues && c.ISV) pack_expand<true>(c, e0, n, key0, tag, set, sink);
            else pack_expand<false>(c, e0, n, key0, tag, set, sink);
        }
        __syncwarp();
        first = end;
    }
}

// Stages (x value, z value) pairs across a warp's packs (see PairStageSink).
struct PackSink {
    static constexpr bool kValues = true;
    uint2* stage;
    uint2* out;
    Reserve rs;
    uint32_t n = 0;
    unsigned long long done = 0;  // pairs flushed

    __device__ __forceinline__ uint32_t tag(const RowCtx& c, uint32_t x) const { return c.id2x[x]; }
    __device__ __forceinline__ void flush() {
        if (n == 0) return;
        done += n;
        unsigned long long base = 0;
        if (lane_id() == 0) base = atomicAdd(rs.cursor, (unsigned long long)n);
        base = __shfl_sync(0xffffffffu, base, 0);
        __syncwarp();
        if (base + n <= rs.cap)
            for (uint32_t i = lane_id(); i < n; i += 32) st_stream(&out[base + i], stage[i]);
        __syncwarp();
        n = 0;
    }
    template <uint32_t N>
    __device__ __forceinline__ void take(const uint32_t (&b)[N], const uint32_t (&x)[N], const uint32_t (&v)[N]) {
        uint32_t tot = 0;
#pragma unroll
        for (uint32_t u = 0; u < N; u++) tot += __popc(b[u]);
        if (tot == 0) return;
        if (n + tot > kPackStage) flush();
        const uint32_t lt = lanemask_lt();
        uint32_t pos = n;
#pragma unroll
        for (uint32_t u = 0; u < N; u++) {
            if (b[u] & (1u << lane_id())) stage[pos + __popc(b[u] & lt)] = make_uint2(x[u], v[u]);
            pos += __popc(b[u]);
        }
        n += tot;
    }
};

// One join's small rows.
static __global__ void __launch_bounds__(256, 4) k_single_pack(RowCtx c, Reserve rs, unsigned long long* cls,
                                                               const uint32_t* __restrict__ rows,
                                                               const unsigned long long* __restrict__ nrows_p) {
    extern __shared__ uint32_t smem[];
    const uint32_t nw = blockDim.x >> 5, wib = threadIdx.x >> 5, lane = lane_id();
    uint32_t* tab = smem + (size_t)wib * kPackWords;
    PackSink sink{reinterpret_cast<uint2*>(tab + (1u << kPackLg)), c.out, rs};
    const uint32_t nrows = (uint32_t)*nrows_p;
    // rows a warp takes at a time: fewer where 32 would leave warps without any
    const uint32_t warps = gridDim.x * nw;
    uint32_t take = (nrows + warps - 1) / warps;
    take = take > 32 ? 32 : take;
    for (uint64_t r0 = (uint64_t)(blockIdx.x * nw + wib) * take; r0 < nrows; r0 += (uint64_t)warps * take) {
        const uint32_t n = (uint32_t)min((uint64_t)take, nrows - r0);
        const uint32_t x = lane < n ? rows[r0 + lane] : 0u;
        pack_rows(c, x, 0, n, tab, sink);
    }
    sink.flush();
    if (lane == 0 && sink.done) atomicAdd(cls, sink.done);
}

}  // namespace dim3g
