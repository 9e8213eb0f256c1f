// noalloc.cu -- join-project for callers that cannot allocate device memory.
//
// Some callers cannot call cudaMalloc at the point where they need a join:
// code running under a custom or fixed-budget allocator that forbids the
// runtime's allocator, real-time or embedded hosts that preallocate
// everything at start-up, and pipelines that must not trigger the implicit
// device synchronisation an allocation can cause.  dim3g_join_project_noalloc
// serves them: it takes device inputs and a caller-provided output buffer,
// and keeps all of its scratch in one file-scope device array of fixed size,
// so it never calls cudaMalloc, cudaFree or any allocating routine.
//
// Costs and limits (stated in include/dim3gpu.h):
//   - every GPU that loads this library holds kScratchBytes (about 20 MB)
//     for the life of the process;
//   - the larger relation may hold at most DIM3G_NOALLOC_MAX_TUPLES tuples
//     and the result at most DIM3G_NOALLOC_MAX_PAIRS distinct pairs;
//   - all calls share the one array, so calls whose work overlaps on the GPU
//     (different streams, different host threads) race and corrupt each
//     other; serialise them.
// The scratch array's name is a host-side stand-in, not a device address;
// the host resolves the real address with cudaGetSymbolAddress, once per
// device, with that device current, on the first call made on that device.
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <mutex>

#include "../../include/dim3gpu.h"

namespace {

constexpr uint32_t kMaxTuples = DIM3G_NOALLOC_MAX_TUPLES;  // larger relation
constexpr uint32_t kMaxPairs = DIM3G_NOALLOC_MAX_PAIRS;    // distinct output pairs
constexpr uint32_t kBuckets = 1u << 17;                     // buckets on the join key
constexpr uint32_t kPairSlots = 2 * kMaxPairs;              // pair set, load factor <= ~1/2
constexpr unsigned long long kEmptyPair = ~0ull;
// The probe's tasks: a run of 32 probe tuples is cut into pieces of at least
// kPiece candidates (as many as the task list has room for), so that a few
// join values with long buckets do not leave their candidates to one warp.
constexpr uint32_t kPiece = 1024, kMaxTasks = kMaxTuples / 32 * 16;
constexpr int kThreads = 512, kCtasPerSm = 3;

// Layout of the scratch array (byte offsets, 256-aligned).  The counters and
// bucket counts are zeroed together.
constexpr size_t kOffCounters = 0;
constexpr size_t kOffCount = kOffCounters + 256;
constexpr size_t kOffBase = kOffCount + (size_t)kBuckets * 4;
constexpr size_t kOffSorted = kOffBase + (size_t)kBuckets * 4;
constexpr size_t kOffTasks = kOffSorted + (size_t)kMaxTuples * 8;
constexpr size_t kOffPairs = kOffTasks + (size_t)kMaxTasks * 4;
constexpr size_t kScratchBytes = kOffPairs + (size_t)kPairSlots * 8;

static __device__ __align__(256) unsigned char g_scratch[kScratchBytes];

struct Counters {
    unsigned long long n_out;    // distinct pairs found
    unsigned long long flags;    // bit 1: a probe walked the whole pair table
    unsigned long long all_ones; // the all-ones pair seen
    uint32_t placed;             // sorted tuples given to buckets
    uint32_t n_tasks, next_task;
};
static_assert(sizeof(Counters) <= 256, "counters' room");

struct Scratch {
    Counters* c;
    uint32_t* count;  // tuples per bucket
    uint32_t* base;   // first sorted tuple of each bucket; its end once placed
    uint2* sorted;    // the larger relation, bucket by bucket
    uint32_t* tasks;  // run of 32 probe tuples * pieces a run + piece
    unsigned long long* pairs;
};

__device__ __forceinline__ uint32_t mix32(uint32_t h) {
    h ^= h >> 16;
    h *= 0x85ebca6bu;
    h ^= h >> 13;
    h *= 0xc2b2ae35u;
    h ^= h >> 16;
    return h;
}
__device__ __forceinline__ unsigned long long mix64(unsigned long long v) {
    v = (v ^ (v >> 30)) * 0xbf58476d1ce4e5b9ull;
    v = (v ^ (v >> 27)) * 0x94d049bb133111ebull;
    return v ^ (v >> 31);
}

__device__ __forceinline__ uint32_t bucket_of(uint32_t y) { return mix32(y) & (kBuckets - 1); }
__device__ __forceinline__ uint32_t lane() { return threadIdx.x & 31; }
__device__ __forceinline__ uint32_t warp_scan(uint32_t v) {  // inclusive
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if ((int)lane() >= o) v += t;
    }
    return v;
}

// Distinct-pair set: 64-bit keys (P.first << 32 | Q.first) with linear
// probing; the all-ones key is tracked by a flag.  `cur`: the key's first
// slot h, already loaded.  True for a pair's first insertion.
__device__ bool insert_pair(const Scratch& s, unsigned long long key, uint32_t h, unsigned long long cur) {
    if (key == kEmptyPair) return atomicExch(&s.c->all_ones, 1ull) == 0ull;
    for (uint32_t p = 0;;) {
        if (cur == key) return false;
        if (cur == kEmptyPair) {
            cur = atomicCAS(&s.pairs[h], kEmptyPair, key);
            if (cur == kEmptyPair) return true;
            if (cur == key) return false;
        }
        if (++p == kPairSlots) break;
        h = (h + 1) & (kPairSlots - 1);
        cur = __ldcg(&s.pairs[h]);
    }
    atomicOr(&s.c->flags, 2ull);
    return false;
}

// The run of 32 probe tuples from q0: the lane's tuple and its bucket.
struct Run {
    uint2 q;
    uint32_t end, len;  // the bucket's end and length
};
__device__ __forceinline__ Run load_run(const uint2* __restrict__ Q, uint32_t nQ, uint32_t q0, const Scratch& s) {
    Run r{make_uint2(0, 0), 0, 0};
    const uint32_t i = q0 + lane();
    if (i < nQ) {
        r.q = __ldg(&Q[i]);
        const uint32_t b = bucket_of(r.q.y);
        r.end = __ldcg(&s.base[b]);
        r.len = __ldcg(&s.count[b]);
    }
    return r;
}

// The join.  The larger relation P is placed bucket by bucket of its join key
// (count, give every bucket a range, place; the ranges are in no order, so no
// prefix sum), then the smaller one, Q, probes: the candidates of 32 probe
// tuples are flattened over a warp, each lane comparing one sorted tuple's key,
// and new pairs take one reservation per group of 128 candidates.
//
// Bound by the latency of dependent accesses.  A linked list per bucket,
// walked by one thread a probe tuple, with a reservation a pair, took 205 us
// in the probe alone for 150K x 90K tuples.  The steps are plain launches, each
// with what does not depend on the one before (150K x 90K tuples: 77 us).  One
// cooperative launch with grid barriers between them took 83, and could only
// start once its whole grid fitted beside whatever else ran on the GPU.
__device__ __forceinline__ uint32_t thread_id() { return blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ uint32_t thread_count() { return gridDim.x * blockDim.x; }

// Counts P's buckets; empties the pair set (the previous call's pairs).
__global__ void __launch_bounds__(kThreads) k_na_count(const uint2* __restrict__ P, uint32_t nP, Scratch s) {
    for (uint32_t i = thread_id(); i < nP; i += thread_count()) atomicAdd(&s.count[bucket_of(__ldg(&P[i]).y)], 1u);
    const uint32_t ones = 0xFFFFFFFFu;
    for (uint32_t i = thread_id(); i < kPairSlots / 2; i += thread_count())
        reinterpret_cast<uint4*>(s.pairs)[i] = make_uint4(ones, ones, ones, ones);
}

// Pieces a run of 32 probe tuples may have.
__device__ __forceinline__ uint32_t most_pieces(uint32_t nQ) { return kMaxTasks / ((nQ + 31) / 32); }

// Ranges: a warp's 128 buckets take one range, four buckets a lane.  Tasks:
// the pieces of every run of 32 probe tuples.
__global__ void __launch_bounds__(kThreads) k_na_ranges(const uint2* __restrict__ Q, uint32_t nQ, Scratch s) {
    const uint32_t warp = thread_id() >> 5, warps = thread_count() >> 5, ln = lane();
    for (uint32_t b0 = warp * 128; b0 < kBuckets; b0 += warps * 128) {
        const uint4 n = reinterpret_cast<const uint4*>(s.count + b0)[ln];
        const uint32_t sum = n.x + n.y + n.z + n.w, inc = warp_scan(sum);
        const uint32_t tot = __shfl_sync(0xffffffffu, inc, 31);
        if (tot == 0) continue;
        uint32_t at = 0;
        if (ln == 0) at = atomicAdd(&s.c->placed, tot);
        at = __shfl_sync(0xffffffffu, at, 0) + inc - sum;
        reinterpret_cast<uint4*>(s.base + b0)[ln] = make_uint4(at, at + n.x, at + n.x + n.y, at + n.x + n.y + n.z);
    }
    const uint32_t runs = (nQ + 31) / 32, most = most_pieces(nQ);
    for (uint32_t r = warp; r < runs; r += warps) {
        const uint32_t i = r * 32 + ln;
        unsigned long long w = i < nQ ? s.count[bucket_of(__ldg(&Q[i]).y)] : 0u;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
        if (w == 0) continue;
        const uint32_t n = (uint32_t)min((w + kPiece - 1) / kPiece, (unsigned long long)most);
        uint32_t at = 0;
        if (ln == 0) at = atomicAdd(&s.c->n_tasks, n);
        at = __shfl_sync(0xffffffffu, at, 0);
        for (uint32_t k = ln; k < n; k += 32) s.tasks[at + k] = r * most + k;
    }
}

// Places P's tuples (base becomes the bucket's end).
__global__ void __launch_bounds__(kThreads) k_na_place(const uint2* __restrict__ P, uint32_t nP, Scratch s) {
    for (uint32_t i = thread_id(); i < nP; i += thread_count()) {
        const uint2 p = __ldg(&P[i]);
        s.sorted[atomicAdd(&s.base[bucket_of(p.y)], 1u)] = p;
    }
}

__global__ void __launch_bounds__(kThreads, kCtasPerSm)
    k_na_join(const uint2* __restrict__ Q, uint32_t nQ, Scratch s, uint2* out, unsigned long long cap) {
    const uint32_t most = most_pieces(nQ), ln = lane(), lt = (1u << ln) - 1u;
    const uint32_t tasks = __ldcg(&s.c->n_tasks);
    for (;;) {
        uint32_t t = 0;
        if (ln == 0) t = atomicAdd(&s.c->next_task, 1u);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= tasks) break;
        const uint32_t task = __ldcg(&s.tasks[t]), piece = task % most;
        const Run run = load_run(Q, nQ, task / most * 32, s);
        // 32 buckets of at most 2^18 tuples: the prefix fits 32 bits
        const uint32_t inc = warp_scan(run.len);
        const uint32_t w = __shfl_sync(0xffffffffu, inc, 31);
        const uint32_t n = min((w + kPiece - 1) / kPiece, most), share = (w + n - 1) / n;
        const uint32_t lo = min(w, piece * share), hi = min(w, lo + share);
        for (uint32_t cb = lo; cb < hi; cb += 128) {
            // a result past the limit is already known: no more pairs are
            // claimed (those in flight fit the table's second half)
            unsigned long long found = 0;
            if (ln == 0) found = *(volatile unsigned long long*)&s.c->n_out;
            if (__shfl_sync(0xffffffffu, found, 0) > kMaxPairs) return;
            uint2 p[4], q[4];
            uint32_t b[4], tot = 0;
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {
                const uint32_t ci = min(cb + u * 32 + ln, hi - 1);
                uint32_t k = 0;  // the probe tuple holding candidate ci
#pragma unroll
                for (uint32_t step = 16; step >= 1; step >>= 1)
                    if (__shfl_sync(0xffffffffu, inc, k + step - 1) <= ci) k += step;
                const uint32_t j = __shfl_sync(0xffffffffu, run.end - inc, k) + ci;
                q[u].x = __shfl_sync(0xffffffffu, run.q.x, k);
                q[u].y = __shfl_sync(0xffffffffu, run.q.y, k);
                p[u] = __ldcg(&s.sorted[j]);
            }
            unsigned long long key[4], cur[4];
            uint32_t h[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {
                key[u] = ((unsigned long long)p[u].x << 32) | q[u].x;
                h[u] = (uint32_t)mix64(key[u]) & (kPairSlots - 1);
                if (p[u].y == q[u].y) cur[u] = __ldcg(&s.pairs[h[u]]);
            }
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {
                const bool fresh = cb + u * 32 + ln < hi && p[u].y == q[u].y && insert_pair(s, key[u], h[u], cur[u]);
                b[u] = __ballot_sync(0xffffffffu, fresh);
                tot += __popc(b[u]);
            }
            if (tot == 0) continue;
            unsigned long long pos = 0;
            if (ln == 0) pos = atomicAdd(&s.c->n_out, (unsigned long long)tot);
            pos = __shfl_sync(0xffffffffu, pos, 0);
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {
                if (b[u] >> ln & 1u) {
                    const unsigned long long at = pos + __popc(b[u] & lt);
                    if (at < cap) out[at] = make_uint2(p[u].x, q[u].x);
                }
                pos += __popc(b[u]);
            }
        }
    }
}

// Per-device scratch address and grid size, resolved once with that device
// current.
std::mutex g_setup_mutex;
std::atomic<unsigned char*> g_base[64];
int g_grid[64];

int scratch_for_device(int dev, unsigned char** base, int* grid) {
    if (dev < 0 || dev >= 64) return DIM3G_ERR_UNSUPPORTED;
    unsigned char* p = g_base[dev].load(std::memory_order_acquire);
    if (!p) {
        std::lock_guard<std::mutex> lock(g_setup_mutex);
        p = g_base[dev].load(std::memory_order_relaxed);
        if (!p) {
            int sms = 0;
            if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) {
                cudaGetLastError();
                return DIM3G_ERR_CUDA;
            }
            void* addr = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&addr, g_scratch);
            if (e != cudaSuccess || !addr) {
                cudaGetLastError();
                return DIM3G_ERR_CUDA;
            }
            g_grid[dev] = sms * kCtasPerSm;
            p = (unsigned char*)addr;
            g_base[dev].store(p, std::memory_order_release);
        }
    }
    *base = p;
    *grid = g_grid[dev];
    return DIM3G_OK;
}

bool aligned8(const void* p) { return ((uintptr_t)p & 7u) == 0; }

}  // namespace

extern "C" int dim3g_join_project_noalloc(const uint32_t* d_R, uint64_t nR, const uint32_t* d_S, uint64_t nS,
                                          uint32_t* d_out, uint64_t capacity, uint64_t* n_out, void* cuda_stream) {
    if (!n_out || (nR && !d_R) || (nS && !d_S) || (capacity && !d_out)) return DIM3G_ERR_INVALID;
    *n_out = 0;
    // the kernels read and write pairs as 8-byte words
    if (!aligned8(d_R) || !aligned8(d_S) || !aligned8(d_out)) return DIM3G_ERR_INVALID;
    // the larger relation drives the build, exactly the reference's swap
    const bool swap = nR < nS;
    const uint2* P = (const uint2*)(swap ? d_S : d_R);
    const uint2* Q = (const uint2*)(swap ? d_R : d_S);
    const uint64_t nP = swap ? nS : nR, nQ = swap ? nR : nS;
    if (nP == 0 || nQ == 0) return DIM3G_OK;            // an empty input joins to nothing
    if (nP > kMaxTuples) return DIM3G_ERR_UNSUPPORTED;  // beyond the fixed scratch
    // An error the caller left pending (from earlier, unrelated work) is
    // reported and left in place, not taken as this call's launch status.
    if (cudaPeekAtLastError() != cudaSuccess) return DIM3G_ERR_CUDA;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return DIM3G_ERR_CUDA;
    }
    unsigned char* base = nullptr;
    int grid = 0;
    int r = scratch_for_device(dev, &base, &grid);
    if (r) return r;
    Scratch s{(Counters*)(base + kOffCounters), (uint32_t*)(base + kOffCount), (uint32_t*)(base + kOffBase),
              (uint2*)(base + kOffSorted), (uint32_t*)(base + kOffTasks), (unsigned long long*)(base + kOffPairs)};
    cudaStream_t st = (cudaStream_t)cuda_stream;
    // the previous call's contents stay in the array: the counters and bucket
    // counts start at zero, k_na_count empties the pair set
    if (cudaMemsetAsync(s.c, 0, kOffBase - kOffCounters, st) != cudaSuccess) {
        cudaGetLastError();
        return DIM3G_ERR_CUDA;
    }
    auto ctas = [&](uint64_t threads) {
        const uint64_t n = (threads + kThreads - 1) / kThreads;
        return (unsigned)(n < (uint64_t)grid ? n : (uint64_t)grid);
    };
    const uint32_t n_p = (uint32_t)nP, n_q = (uint32_t)nQ;
    k_na_count<<<(unsigned)grid, kThreads, 0, st>>>(P, n_p, s);
    k_na_ranges<<<ctas(nQ > kBuckets / 4 ? nQ : kBuckets / 4), kThreads, 0, st>>>(Q, n_q, s);
    k_na_place<<<ctas(nP), kThreads, 0, st>>>(P, n_p, s);
    // the candidates are not known: at least a CTA an SM
    const unsigned c_join = ctas(nP + nQ), c_sm = (unsigned)(grid / kCtasPerSm);
    k_na_join<<<c_join > c_sm ? c_join : c_sm, kThreads, 0, st>>>(Q, n_q, s, (uint2*)d_out, capacity);
    unsigned long long h[2] = {0, 0};  // n_out, flags
    if (cudaGetLastError() != cudaSuccess || cudaMemcpyAsync(h, s.c, sizeof h, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
        cudaGetLastError();
        return DIM3G_ERR_CUDA;
    }
    if (h[0] > kMaxPairs) return DIM3G_ERR_UNSUPPORTED;  // more distinct pairs than DIM3G_NOALLOC_MAX_PAIRS
    if (h[1]) return DIM3G_ERR_DEVICE;
    *n_out = h[0];
    return h[0] > capacity ? DIM3G_ERR_CAPACITY : DIM3G_OK;
}
