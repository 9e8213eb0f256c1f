// scan.cuh -- device-wide exclusive prefix sums in one launch, driven by
// functors so one pass both computes and consumes the prefix (CSR row
// pointers, table compaction, output offsets).
//
// Decoupled look-back: tiles are numbered by a ticket, so a tile waits only
// on tiles whose CTAs already run.  A tile publishes its sum, adds up its
// predecessors' published words 32 at a time back to the nearest inclusive
// prefix, and publishes its own.  Items are read once and a scan is one
// launch.  (Sum of tiles, scan of the sums, apply -- three launches and two
// reads -- were 45 of the 53 kernels of a small join, at about 3 us each.)
#pragma once
#include "common.cuh"

namespace dim3g {

constexpr int kScanBlock = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanBlock * kScanItems;
// Values below this add up to less than 2^32 in a tile (a power of two: so do
// values whose bits taken together are).
constexpr uint32_t kScanNarrow = (uint32_t)((1ull << 32) / kScanTile);

// A tile's word: sum << 2 | state (sums stay below 2^62).
constexpr unsigned long long kScanSum = 1, kScanPrefix = 2;
// Polls of one look-back window before a tile gives up (about a second).
constexpr uint32_t kScanPolls = 1u << 21;

// One scan.  Src: uint32_t operator()(i), the value of item i, i < n, and
// Src::Sum, the type that a tile's values are added up in: uint32_t where 4096
// consecutive ones stay below 2^32 (0/1 flags, and counts of the tuples of a
// relation, which holds fewer), else uint64_t.
// Dst: void operator()(i, prefix, value).  state: scan_storage(n) zeroed
// words.  *total (may be null) receives the sum.  lim (may be null): the
// length where only the device knows it (the launch covers the host's bound
// n; tiles at or past *lim end at once).
template <class Src, class Dst>
struct ScanJob {
    Src src;
    Dst dst;
    uint64_t n;
    unsigned long long* state;
    unsigned long long* total;
    const unsigned long long* lim = nullptr;
};

inline uint64_t scan_blocks(uint64_t n) { return (n + kScanTile - 1) / kScanTile; }
inline uint64_t scan_storage(uint64_t n) { return scan_blocks(n) + 1; }

// Exclusive prefix of tile `tile` (its sum: `sum`), by one warp.
__device__ __forceinline__ uint64_t scan_look_back(unsigned long long* state, uint64_t tile, uint64_t sum,
                                                   uint32_t* err) {
    volatile unsigned long long* w = state + 1;
    const uint32_t lane = lane_id();
    if (tile == 0) {
        if (lane == 0) w[0] = sum << 2 | kScanPrefix;
        return 0;
    }
    if (lane == 0) w[tile] = sum << 2 | kScanSum;
    uint64_t before = 0;
    for (uint64_t end = tile;; end -= 32) {  // lane l reads tile end - 1 - l
        unsigned long long v = kScanPrefix;
        uint32_t polls = 0;
        for (;;) {
            if (lane < end) v = w[end - 1 - lane];
            if (__all_sync(0xffffffffu, (v & 3) != 0)) break;
            if (++polls == kScanPolls) {
                if (lane == 0) raise_error(err, kErrScanTimeout);
                break;
            }
        }
        const uint32_t done = __ballot_sync(0xffffffffu, (v & 3) == kScanPrefix);
        const uint32_t last = done ? __ffs(done) - 1 : 31;
        before += warp_sum<uint64_t>(lane <= last ? v >> 2 : 0ull);
        if (done || polls == kScanPolls || end <= 32) break;
    }
    if (lane == 0) w[tile] = (before + sum) << 2 | kScanPrefix;
    return before;
}

// Values v of a tile, sums in Sum: the prefix of each to dst.  A warp owns
// 32 x kScanItems consecutive items, lane l of step k the item 32 k + l, so
// loads and stores are coalesced; the prefixes of a step come from a warp
// scan.  (kScanItems consecutive items a thread made every store of a warp
// touch 32 sectors.)
template <class Sum, class Src, class Dst>
__device__ __forceinline__ void scan_tile(const ScanJob<Src, Dst>& j, const uint32_t (&v)[kScanItems], uint64_t first,
                                          uint64_t n, uint64_t tile, uint64_t nb, uint32_t* err, uint32_t lane, uint32_t wib) {
    constexpr int kWarps = kScanBlock / 32;
    __shared__ Sum s_warp[kWarps];
    __shared__ uint64_t s_before;
    Sum e[kScanItems], run = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        const Sum inc = warp_incl_scan<Sum>(v[k]);
        e[k] = run + inc - v[k];
        run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) s_warp[wib] = run;
    __syncthreads();
    if (wib == 0) {
        const Sum t = lane < kWarps ? s_warp[lane] : Sum(0);
        const Sum inc = warp_incl_scan(t);
        const uint64_t sum = __shfl_sync(0xffffffffu, inc, kWarps - 1);
        if (lane < kWarps) s_warp[lane] = inc - t;
        const uint64_t before = scan_look_back(j.state, tile, sum, err);
        if (lane == 0) {
            s_before = before;
            if (tile == nb - 1 && j.total) *j.total = before + sum;
        }
    }
    __syncthreads();
    const uint64_t at = s_before + s_warp[wib];
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        const uint64_t i = first + 32 * k;
        if (i < n) j.dst(i, at + e[k], v[k]);
    }
}

// Up to two scans of one kind (blockIdx.y) in one launch.  64-bit sums only
// in tiles that can pass 2^32: the wider warp scans take twice the time (86K
// row counts: 13.6 us in 64 bits, 6.1 in 32).
template <class Src, class Dst>
__global__ void __launch_bounds__(kScanBlock) k_scan(ScanJob<Src, Dst> a, ScanJob<Src, Dst> b, uint32_t* err) {
    __shared__ uint64_t s_tile;
    const ScanJob<Src, Dst> j = blockIdx.y ? b : a;
    const uint64_t n = j.lim && *j.lim < j.n ? *j.lim : j.n;
    const uint64_t nb = (n + kScanTile - 1) / kScanTile;
    if (blockIdx.x >= nb) return;
    if (threadIdx.x == 0) s_tile = atomicAdd(j.state, 1ull);
    __syncthreads();
    const uint64_t tile = s_tile;
    const uint32_t lane = lane_id(), wib = threadIdx.x >> 5;
    const uint64_t first = tile * kScanTile + wib * (32 * kScanItems) + lane;
    uint32_t v[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        const uint64_t i = first + 32 * k;
        v[k] = i < n ? (uint32_t)j.src(i) : 0u;
    }
    if constexpr (sizeof(typename Src::Sum) > 4) {
        uint32_t bits = 0;
#pragma unroll
        for (int k = 0; k < kScanItems; k++) bits |= v[k];
        if (__syncthreads_or(bits >= kScanNarrow)) {
            scan_tile<uint64_t>(j, v, first, n, tile, nb, err, lane, wib);
            return;
        }
    }
    scan_tile<uint32_t>(j, v, first, n, tile, nb, err, lane, wib);
}

// Host launches; the states are zeroed by the caller.  An empty scan launches
// nothing and leaves *total as it is (zeroed with the rest).
template <class Src, class Dst>
inline void device_scan(const ScanJob<Src, Dst>& j, uint32_t* err, cudaStream_t st) {
    if (j.n) k_scan<<<(unsigned)scan_blocks(j.n), kScanBlock, 0, st>>>(j, j, err);
}
template <class Src, class Dst>
inline void device_scan2(const ScanJob<Src, Dst>& a, const ScanJob<Src, Dst>& b, uint32_t* err, cudaStream_t st) {
    const uint64_t n = a.n > b.n ? a.n : b.n;
    if (n) k_scan<<<dim3((unsigned)scan_blocks(n), 2), kScanBlock, 0, st>>>(a, b, err);
}

}  // namespace dim3g
