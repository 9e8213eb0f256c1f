// mapping.cuh -- value -> dense id mapping on the GPU (the role of the
// reference's mapping_step + LS_mapper, dim3.hpp:394-883 and
// Include/L+S_mapper.hpp:11-160), plus the CSR builds (divide_R
// dim3.hpp:1058-1086, the sparse half of divide_S dim3.hpp:1186-1253).
//
// Table layout: one 64-bit slot per entry, key in the high half, dense id in
// the low half; the all-ones word marks an empty slot, so every 32-bit key
// (0xFFFFFFFF included) is a valid key.  Open addressing with linear probing
// at load factor <= 1/2; ids are assigned after the build by a prefix sum
// over occupied slots, so they are dense in [0, count).
#pragma once
#include "common.cuh"
#include "scan.cuh"

namespace dim3g {

constexpr uint32_t kNotFound = 0xFFFFFFFFu;

struct DevTable {
    unsigned long long* slots;
    uint64_t mask;       // capacity - 1 (capacity is a power of two)
    uint64_t limit = 0;  // longest probe (0: the whole table)
};

__device__ __forceinline__ bool table_insert(DevTable t, uint32_t key, uint32_t* err) {
    uint64_t h = mix32(key) & t.mask;
    const unsigned long long want = (unsigned long long)key << 32;
    const uint64_t lim = t.limit ? t.limit : t.mask;
    for (uint64_t p = 0; p <= lim; p++) {
        unsigned long long cur = __ldcg(&t.slots[h]);
        if (cur == kEmpty64) {
            unsigned long long prev = atomicCAS(&t.slots[h], (unsigned long long)kEmpty64, want);
            if (prev == kEmpty64) return true;
            cur = prev;
        }
        if ((uint32_t)(cur >> 32) == key) return false;
        h = (h + 1) & t.mask;
    }
    raise_error(err, kErrProbeLimit);
    return false;
}

__device__ __forceinline__ uint32_t table_find(DevTable t, uint32_t key) {
    uint64_t h = mix32(key) & t.mask;
    const uint64_t lim = t.limit ? t.limit : t.mask;
    for (uint64_t p = 0; p <= lim; p++) {
        unsigned long long cur = __ldg(&t.slots[h]);
        if (cur == kEmpty64) return kNotFound;
        if ((uint32_t)(cur >> 32) == key) return (uint32_t)cur;
        h = (h + 1) & t.mask;
    }
    return kNotFound;
}

// Tuples a thread of the sketch pass holds in flight.
constexpr uint32_t kMapIlp = 4;

// Table sizing.  A table built for a relation's tuple count (load factor
// 1/2 if every key were distinct) is far larger than its distinct keys when
// keys repeat -- 2^26 slots, 512 MB, for the 2M vertices of a 20M-edge graph
// -- and every insert and probe then misses the L2.  A HyperLogLog sketch
// (2^kSketchLg registers, one pass, about 2.3 % standard error) of the three
// key columns sizes each table to about 1.5x its distinct keys instead.
// Probes of a sketch-sized table are bounded by kSizedProbeLimit; a build
// that exceeds it (a table fuller than the sketch said) is redone with the
// tuple-sized tables, so the result never depends on the estimate.
constexpr uint32_t kSketchLg = 11, kSketchRegs = 1u << kSketchLg;
constexpr uint64_t kSizedProbeLimit = 1u << 12;

// A key's register (the hash's top kSketchLg bits) and rank (leading zeros
// of the rest, plus one).
__device__ __forceinline__ uint2 sketch_slot(uint32_t key) {
    const unsigned long long h = mix64((unsigned long long)key + 0x9E3779B97F4A7C15ull);
    const unsigned long long w = h << kSketchLg;
    return make_uint2((uint32_t)(h >> (64 - kSketchLg)), (w ? (uint32_t)__clzll(w) : 64u - kSketchLg) + 1);
}

inline uint64_t next_pow2(uint64_t v) {
    uint64_t p = 1;
    while (p < v) p <<= 1;
    return p;
}

// Adds a key: no atomic when the register already holds the rank (most
// updates once the registers have filled).
__device__ __forceinline__ void sketch_add_if_larger(uint32_t* r, uint32_t key) {
    const uint2 s = sketch_slot(key);
    if (*(volatile uint32_t*)&r[s.x] < s.y) atomicMax(&r[s.x], s.y);
}

// HyperLogLog estimate (with the small-range correction) from a column's
// register sum (sum of 2^-r) and count of zero registers; the table slots for
// it, slack_pct slots per estimated key, a power of two no larger than full.
inline double sketch_estimate(double sum, uint32_t zeros) {
    const double M = kSketchRegs;
    double e = 0.7213 / (1.0 + 1.079 / M) * M * M / sum;
    if (e <= 2.5 * M && zeros) e = M * log(M / zeros);
    return e;
}
inline uint64_t sketch_capacity(double est, uint64_t full, uint32_t slack_pct) {
    const uint64_t cap = next_pow2((uint64_t)(slack_pct / 100.0 * est) + 1024);
    return cap < full ? cap : full;
}

// Registers of P's first and y columns and Q's first column, kSketchRegs
// each, merged into regs (zeroed by the caller).  Bound by the latency of the
// tuple loads, so kMapIlp of them are in flight a thread, at
// kSketchThreads x 4 threads an SM; a CTA's registers are merged with an
// atomic only where they raise the total (few do once the first CTAs have
// merged).  2 x 10M tuples: 151 us at 256 x 2 threads an SM and one load in
// flight.
constexpr int kSketchThreads = 512;
static __global__ void __launch_bounds__(kSketchThreads) k_sketch(const uint2* __restrict__ P, uint64_t nP,
                                                                  const uint2* __restrict__ Q, uint64_t nQ,
                                                                  uint32_t* regs) {
    __shared__ uint32_t r[3 * kSketchRegs];
    for (uint32_t k = threadIdx.x; k < 3 * kSketchRegs; k += blockDim.x) r[k] = 0;
    __syncthreads();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (uint64_t i = first; i < nP; i += kMapIlp * stride) {
        uint2 p[kMapIlp];
#pragma unroll
        for (uint32_t k = 0; k < kMapIlp; k++)
            if (i + k * stride < nP) p[k] = __ldg(&P[i + k * stride]);
#pragma unroll
        for (uint32_t k = 0; k < kMapIlp; k++)
            if (i + k * stride < nP) {
                sketch_add_if_larger(r, p[k].x);
                sketch_add_if_larger(r + kSketchRegs, p[k].y);
            }
    }
    for (uint64_t i = first; i < nQ; i += kMapIlp * stride) {
        uint32_t q[kMapIlp];
#pragma unroll
        for (uint32_t k = 0; k < kMapIlp; k++)
            if (i + k * stride < nQ) q[k] = __ldg(&Q[i + k * stride].x);
#pragma unroll
        for (uint32_t k = 0; k < kMapIlp; k++)
            if (i + k * stride < nQ) sketch_add_if_larger(r + 2 * kSketchRegs, q[k]);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < 3 * kSketchRegs; k += blockDim.x)
        if (r[k] > __ldcg(&regs[k])) atomicMax(&regs[k], r[k]);
}

// Build pass over the larger relation P: insert its first column into tx and
// its y column into ty.
static __global__ void k_insert_p(const uint2* __restrict__ P, uint64_t n, DevTable tx, DevTable ty, uint32_t* err) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint2 p = P[i];
        table_insert(tx, p.x, err);
        table_insert(ty, p.y, err);
    }
}

// Semi-join of Q against ty (mapping_y's probe, dim3.hpp:816-827): keep the
// tuples whose y occurs in P as (c, y id), insert their first column into tz.
// The kept tuples of a CTA's kProbeItems x 256 tuples take one range of Qk:
// one atomic on the shared counter per 1024 tuples.  (One per warp and 32
// tuples serialised on its address: 431 us for 10M tuples, 893 us for 20M.)
constexpr uint32_t kProbeItems = 4;
static __global__ void __launch_bounds__(256) k_probe_q(const uint2* __restrict__ Q, uint64_t n, DevTable ty,
                                                        DevTable tz, uint2* __restrict__ Qk, unsigned long long* nkept,
                                                        uint32_t* err) {
    __shared__ uint32_t s_cnt[8];
    __shared__ unsigned long long s_base;
    const uint32_t wib = threadIdx.x >> 5, lt = lanemask_lt();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x; i0 < n; i0 += kProbeItems * stride) {
        uint2 q[kProbeItems];
        uint32_t yid[kProbeItems], b[kProbeItems], cnt = 0;
#pragma unroll
        for (uint32_t k = 0; k < kProbeItems; k++) {
            const uint64_t i = i0 + k * stride + threadIdx.x;
            if (i < n) q[k] = __ldg(&Q[i]);
        }
#pragma unroll
        for (uint32_t k = 0; k < kProbeItems; k++) {
            yid[k] = kNotFound;
            if (i0 + k * stride + threadIdx.x < n) {
                yid[k] = table_find(ty, q[k].y);
                if (yid[k] != kNotFound) table_insert(tz, q[k].x, err);
            }
        }
        __syncwarp();
#pragma unroll
        for (uint32_t k = 0; k < kProbeItems; k++) {
            b[k] = __ballot_sync(0xffffffffu, yid[k] != kNotFound);
            cnt += __popc(b[k]);
        }
        if (lane_id() == 0) s_cnt[wib] = cnt;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t t = 0;
            for (uint32_t w = 0; w < 8; w++) {
                const uint32_t c = s_cnt[w];
                s_cnt[w] = t;
                t += c;
            }
            s_base = t ? atomicAdd(nkept, (unsigned long long)t) : 0ull;
        }
        __syncthreads();
        unsigned long long pos = s_base + s_cnt[wib];
#pragma unroll
        for (uint32_t k = 0; k < kProbeItems; k++) {
            if (yid[k] != kNotFound) Qk[pos + __popc(b[k] & lt)] = make_uint2(q[k].x, yid[k]);
            pos += __popc(b[k]);
        }
        __syncthreads();  // s_cnt and s_base are rewritten by the next round
    }
}

// Table compaction: ids by prefix sum over occupied slots.
struct OccupiedSrc {
    using Sum = uint32_t;
    const unsigned long long* slots;
    __device__ uint64_t operator()(uint64_t i) const { return slots[i] != kEmpty64 ? 1u : 0u; }
};
struct AssignIdDst {
    unsigned long long* slots;
    uint32_t* id2v;
    __device__ void operator()(uint64_t i, uint64_t e, uint64_t v) const {
        if (!v) return;
        unsigned long long s = slots[i];
        uint32_t key = (uint32_t)(s >> 32);
        slots[i] = ((unsigned long long)key << 32) | (uint32_t)e;
        if (id2v) id2v[e] = key;
    }
};

// P -> (x id, y id) with the per-x degree histogram (blockIdx.y 0), and Q' =
// (z value, y id) -> z id with the histogram over the (y, z tile) CSR key
// y*T + z/TB (blockIdx.y 1): independent passes in one launch, so the one's
// tail overlaps the other.
struct MapArgs {
    const uint2* P;
    uint64_t nP;
    DevTable tx, ty;
    uint2* Pm;
    uint32_t* degx;
    const uint2* Qk;
    uint64_t nQ;  // kept tuples, or a bound on them with the count in *nkept
    const unsigned long long* nkept;
    DevTable tz;
    uint32_t T, tile_shift;
    uint32_t* zid;
    uint32_t* cnt_yt;
};
static __global__ void __launch_bounds__(256) k_map(MapArgs a) {
    const uint64_t first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    if (blockIdx.y == 0) {
        for (uint64_t i = first; i < a.nP; i += stride) {
            const uint2 p = __ldg(&a.P[i]);
            const uint32_t xi = table_find(a.tx, p.x);
            const uint32_t yi = table_find(a.ty, p.y);
            a.Pm[i] = make_uint2(xi, yi);
            atomicAdd(&a.degx[xi], 1u);
        }
    } else {
        const uint64_t nQ = a.nkept ? *a.nkept : a.nQ;
        for (uint64_t i = first; i < nQ; i += stride) {
            const uint2 q = __ldg(&a.Qk[i]);
            const uint32_t zi = table_find(a.tz, q.x);
            a.zid[i] = zi;
            atomicAdd(&a.cnt_yt[(uint64_t)q.y * a.T + (zi >> a.tile_shift)], 1u);
        }
    }
}

// Row pointers from a histogram: JR[i] = cursor[i] = exclusive prefix.
struct U32Src {
    using Sum = uint32_t;
    const uint32_t* a;
    __device__ uint64_t operator()(uint64_t i) const { return a[i]; }
};
struct RowPtrDst {
    uint32_t* jr;
    uint32_t* cursor;
    __device__ void operator()(uint64_t i, uint64_t e, uint64_t) const {
        jr[i] = (uint32_t)e;
        cursor[i] = (uint32_t)e;
    }
};

// The CSR entries (launched as k_map): R's y ids by x (blockIdx.y 0), and S by
// (y id, z tile) (blockIdx.y 1): z ids (ic_s), and for the expansion paths
// that emit values the z id and z value of each entry side by side (isv; one
// 8-byte load or copy per candidate).  Either may be null: every scattered
// store is a sector of its own, and the pass is bound by those, so a path
// gets only the form that it reads (both 477 us for 10M tuples a side).
struct ScatterArgs {
    const uint2* Pm;
    uint64_t nP;
    uint32_t* curx;
    uint32_t* ic_r;
    const uint2* Qk;
    const uint32_t* zid;
    uint64_t nQ;
    const unsigned long long* nkept;
    uint32_t T, tile_shift;
    uint32_t* cur_yt;
    uint32_t* ic_s;
    uint2* isv;
};
static __global__ void __launch_bounds__(256) k_scatter(ScatterArgs a) {
    const uint64_t first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    if (blockIdx.y == 0) {
        for (uint64_t i = first; i < a.nP; i += stride) {
            const uint2 p = __ldg(&a.Pm[i]);
            a.ic_r[atomicAdd(&a.curx[p.x], 1u)] = p.y;
        }
    } else {
        const uint64_t nQ = a.nkept ? *a.nkept : a.nQ;
        for (uint64_t i = first; i < nQ; i += stride) {
            const uint2 q = __ldg(&a.Qk[i]);
            const uint32_t zi = __ldg(&a.zid[i]);
            const uint32_t pos = atomicAdd(&a.cur_yt[(uint64_t)q.y * a.T + (zi >> a.tile_shift)], 1u);
            if (a.ic_s) a.ic_s[pos] = zi;
            if (a.isv) a.isv[pos] = make_uint2(zi, q.x);
        }
    }
}

}  // namespace dim3g
