// ordered.cuh -- the two-pass form of the row kernels: a count pass writes
// cnt[x] = |distinct z| of every row, a prefix sum over cnt gives the rows'
// offsets, and the write pass repeats the expansion and puts the pairs of row
// x at off[x] on, so rows come in x-id order and each row's pairs together.
// It serves ordered output, counting without output, and callers that size
// their output first.  Same rows, sets and walks as the single pass.
#pragma once
#include "common.cuh"
#include "expand.cuh"
#include "packed.cuh"
#include "single.cuh"

namespace dim3g {

// The sink of a CTA row, and the row's count once its warps are done
// (*s_count is 0 before the row and holds the pairs after it).
template <bool WRITE>
struct RowSink;
template <>
struct RowSink<false> : CountSink {
    __device__ __forceinline__ RowSink(const RowCtx&, uint32_t, uint32_t*) {}
    __device__ __forceinline__ void done(const RowCtx& c, uint32_t x, uint32_t* s_count) {
        if (lane_id() == 0 && count) atomicAdd(s_count, count);
        __syncthreads();
        if (threadIdx.x == 0) c.cnt[x] = *s_count;
    }
};
template <>
struct RowSink<true> : WriteSink {
    __device__ __forceinline__ RowSink(const RowCtx& c, uint32_t x, uint32_t* s_count)
        : WriteSink{c.out, c.err, c.off[x], c.cnt[x], c.id2x[x], s_count} {}
    __device__ __forceinline__ void done(const RowCtx&, uint32_t, uint32_t*) {}
};

// Class 2: one CTA per row, 2^lg table words; the rows as k_single_block's.
template <bool WRITE>
static __global__ void __launch_bounds__(1024, 1) k_rows_block(RowCtx c, const uint32_t* __restrict__ rows,
                                                            const unsigned long long* __restrict__ nrows_p, uint32_t lg,
                                                            const unsigned long long* skip0,
                                                            const unsigned long long* skip1, uint32_t ctr) {
    extern __shared__ uint32_t smem[];
    __shared__ uint32_t s_count, s_row;
    __shared__ CtaChunks s_cc;
    if (threadIdx.x == 0) s_cc.n = 0;
    const uint32_t nrows = (uint32_t)*nrows_p;
    rows += (skip0 ? *skip0 : 0ull) + (skip1 ? *skip1 : 0ull);
    for (uint32_t ri = cta_next_row(&c.next_row[ctr], &s_row); ri < nrows; ri = cta_next_row(&c.next_row[ctr], &s_row)) {
        const uint32_t x = rows[ri];
        if (threadIdx.x == 0) s_count = 0;  // read after the row's first barrier
        RowSink<WRITE> sink(c, x, &s_count);
        single_block_row(c, x, smem, sink, lg, &s_cc);
        sink.done(c, x, &s_count);
    }
}

// Classes 3 and 4: one CTA per row, a bitmap over one z tile at a time; nrows
// = *n4 + *n3, the class-4 rows first.
template <bool WRITE>
static __global__ void __launch_bounds__(1024, 1) k_rows_bitmap(RowCtx c, const uint32_t* __restrict__ rows,
                                                             const unsigned long long* __restrict__ n3,
                                                             const unsigned long long* __restrict__ n4) {
    extern __shared__ uint32_t bm[];
    __shared__ uint32_t s_count, s_row;
    __shared__ CtaChunks s_cc;
    if (threadIdx.x == 0) s_cc.n = 0;
    const uint32_t nrows = (uint32_t)(*n3 + *n4);
    for (uint32_t ri = cta_next_row(&c.next_row[3], &s_row); ri < nrows; ri = cta_next_row(&c.next_row[3], &s_row)) {
        const uint32_t x = rows[ri];
        if (threadIdx.x == 0) s_count = 0;
        RowSink<WRITE> sink(c, x, &s_count);
        single_bitmap_row(c, x, bm, sink, &s_cc);
        sink.done(c, x, &s_count);
    }
}

// Class 1: one warp per row, 2^warp_lg table words per warp.
template <bool WRITE>
static __global__ void __launch_bounds__(256) k_rows_warp(RowCtx c, const uint32_t* __restrict__ rows,
                                                          const unsigned long long* __restrict__ nrows_p,
                                                          uint32_t warp_lg) {
    extern __shared__ uint32_t smem[];
    const uint32_t nw = blockDim.x >> 5, wib = threadIdx.x >> 5, lane = lane_id();
    uint32_t* tab = smem + ((size_t)wib << warp_lg);
    const uint32_t nrows = (uint32_t)*nrows_p;
    for (uint32_t ri = blockIdx.x * nw + wib; ri < nrows; ri += gridDim.x * nw) {
        const uint32_t x = rows[ri];
        if (WRITE) {
            WriteSink sink{c.out, c.err, c.off[x], c.cnt[x], 0, nullptr};
            single_warp_row(c, x, tab, sink, warp_lg);
        } else {
            struct : CountSink {
                uint32_t xv;
            } sink;
            single_warp_row(c, x, tab, sink, warp_lg);
            if (lane == 0) c.cnt[x] = sink.count;
        }
    }
}

// Tiny rows, many to a warp: the pack's candidates carry the lane of their
// row, whose count (or next place) is a shared counter.  A place past the row's
// count is not written.
constexpr size_t kRowsPackWords = ((size_t)1 << kPackLg) + 160;  // table, then a row's counter, value, offset and count
template <bool WRITE>
struct PackRowSink {
    static constexpr bool kValues = WRITE;
    uint32_t* pos;  // 32 counters, 32 first values, 32 offsets (two words each), 32 counts
    uint2* out;
    uint32_t* err;
    __device__ __forceinline__ uint32_t tag(const RowCtx&, uint32_t) const { return lane_id(); }
    template <uint32_t N>
    __device__ __forceinline__ void take(const uint32_t (&b)[N], const uint32_t (&r)[N], const uint32_t (&v)[N]) {
#pragma unroll
        for (uint32_t u = 0; u < N; u++)
            if (b[u] >> lane_id() & 1u) {
                const uint32_t p = atomicAdd(&pos[r[u]], 1u);
                if (WRITE) {
                    const unsigned long long off = reinterpret_cast<const unsigned long long*>(pos + 64)[r[u]];
                    if (p < pos[128 + r[u]]) st_stream(&out[off + p], make_uint2(pos[32 + r[u]], v[u]));
                    else raise_error(err, kErrOutputBound);
                }
            }
    }
};

template <bool WRITE>
static __global__ void __launch_bounds__(256, 4) k_rows_pack(RowCtx c, const uint32_t* __restrict__ rows,
                                                             const unsigned long long* __restrict__ nrows_p) {
    extern __shared__ uint32_t smem[];
    const uint32_t nw = blockDim.x >> 5, wib = threadIdx.x >> 5, lane = lane_id();
    uint32_t* tab = smem + (size_t)wib * kRowsPackWords;
    PackRowSink<WRITE> sink{tab + (1u << kPackLg), c.out, c.err};
    const uint32_t nrows = (uint32_t)*nrows_p, warps = gridDim.x * nw;
    uint32_t take = (nrows + warps - 1) / warps;
    take = take > 32 ? 32 : take;
    for (uint64_t r0 = (uint64_t)(blockIdx.x * nw + wib) * take; r0 < nrows; r0 += (uint64_t)warps * take) {
        const uint32_t n = (uint32_t)min((uint64_t)take, nrows - r0);
        const uint32_t x = lane < n ? rows[r0 + lane] : 0u;
        sink.pos[lane] = 0;
        if (WRITE && lane < n) {
            sink.pos[32 + lane] = c.id2x[x];
            reinterpret_cast<unsigned long long*>(sink.pos + 64)[lane] = c.off[x];
            sink.pos[128 + lane] = c.cnt[x];
        }
        __syncwarp();
        pack_rows(c, x, 0, n, tab, sink);
        if (!WRITE && lane < n) c.cnt[x] = sink.pos[lane];
        if (WRITE && lane < n && sink.pos[lane] != sink.pos[128 + lane]) raise_error(c.err, kErrOutputBound);
        __syncwarp();
    }
}

}  // namespace dim3g
