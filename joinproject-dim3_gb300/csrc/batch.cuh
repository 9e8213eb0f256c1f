// batch.cuh -- many joins per launch.
//
// Relation set: for every relation r of a set (tuples (f, y), f the first
// column) one segmented pass builds, for all relations at once,
//   TF, TY      value -> id tables (f and y), ids dense per relation
//   CSR by f    JRf over the global f-id space, ICf = global y ids
//               (the relation in the role of R)
//   CSR by (y, f tile)  JRy over a per-relation key space y*T + tile (plus
//               T empty sentinel keys), ICy = local f ids, VSy = f values
//               beside them (the relation in the role of S)
// Every relation's ids and keys are local; the set lays them out
// relation-major, so one prefix sum over a whole pool gives every
// relation's CSR at once (a relation's first global position is the tuple
// count of the relations before it).
//
// Query set: joins (P, Q) of relations of a set.  Per query a y map (P's y
// ids -> Q's y ids, or Q's empty sentinel row), P's CSR re-expressed in Q's
// y ids, per-row work and classes; then the row kernels of the single
// relation path run over the rows of all queries, each row fetching its
// query's context.  Kernels take their segment offsets from device memory,
// so a fixed launch sequence (capturable in a CUDA graph) serves any batch
// of a given shape.
#pragma once
#include "aggregate.cuh"
#include "common.cuh"
#include "expand.cuh"
#include "mapping.cuh"
#include "packed.cuh"
#include "single.cuh"

namespace dim3g {

// Largest s in [0, n) with off[s] <= i (off[0..n] nondecreasing, off[0] = 0,
// i < off[n]): the segment holding element i, skipping empty segments.
__device__ __forceinline__ uint32_t seg_find(const uint64_t* __restrict__ off, uint32_t n, uint64_t i) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&off[mid]) <= i) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Per-thread cached segment lookup for loops over contiguous elements.
struct SegCursor {
    const uint64_t* off;
    uint32_t n;
    uint32_t s = 0;
    uint64_t lo = 1, hi = 0;
    __device__ __forceinline__ uint32_t at(uint64_t i) {
        if (i < lo || i >= hi) {
            s = seg_find(off, n, i);
            lo = __ldg(&off[s]);
            hi = __ldg(&off[s + 1]);
        }
        return s;
    }
};

// Grid-ordered element ranges: in round k CTA b takes the elements
// [(k * G + b) * blockDim, + blockDim), G the grid, so the whole grid works
// inside a window of about G * blockDim consecutive elements that moves
// through the relations in order.  The random-address updates of the index
// build (table slots, degree and cursor atomics, the CSR scatter) then fall
// in the few relations under the window, whose tables and CSR slices stay in
// L2, instead of in all of the set at once (CTA-contiguous ranges put the
// grid's CTAs in as many different relations).  The segment of an element is
// looked up again when a thread's next element lies in another relation.
#define DIM3G_FOR_CHUNK(i, n) \
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += (uint64_t)gridDim.x * blockDim.x)

// ------------------------------------------------------------ relation set
struct RelIn {
    const uint2* pairs;  // (f, y) tuples, device
    uint64_t n;
};

// Per-relation layout, computed on the device once the id counts are known.
struct RelDev {
    uint64_t nt;        // tuples
    uint64_t tup_off;   // first position in the tuple-indexed pools
    uint64_t tab_off;   // first slot in TF / TY
    uint64_t tab_cap;   // slots per table (power of two)
    uint64_t nf, ny;    // distinct f, distinct y
    uint64_t fbase, ybase;  // first global f id / y id
    uint64_t yt_base;   // first key of the (y, f tile) key space
    uint32_t T, tile_shift, tile_width;
    uint32_t probe_lim; // longest probe of the tables (0: the whole table)
};

// The CSRs a relation's queries read: kRoleRows, by first value (the
// relation drives the rows of a join); kRoleCols, by (y, z tile) (its first
// values are a join's output column).
enum RelRole : uint8_t { kRoleRows = 1, kRoleCols = 2 };

// Pools of one relation set (device pointers).
struct RelPools {
    const RelIn* in;
    RelDev* rel;
    const uint64_t* tup_off;  // nrel + 1
    const uint64_t* tab_off;  // nrel + 1
    uint32_t nrel;
    uint32_t probe_lim;       // sketch-sized tables: longest probe (0: tuple-sized tables)
    uint64_t ntot;            // sum of tuples
    unsigned long long* TF;
    unsigned long long* TY;
    unsigned long long* nf_cnt;  // nrel
    unsigned long long* ny_cnt;  // nrel
    unsigned long long* tabF;    // occupied slots of TF before every kTabMark-th, and in all
    unsigned long long* tabY;
    uint64_t tab_marks;
    uint32_t* id2f;           // by global f id
    uint32_t* id2y;           // by global y id
    uint2* Pm;                // (global f id, global y id) per tuple
    uint32_t* degF;           // ntot + 1
    uint32_t* JRf;            // ntot + 1, global positions
    uint32_t* curF;
    uint32_t* ICf;            // global y ids
    uint32_t* cnt_yt;         // yt_cap
    uint32_t* JRy;            // yt_cap, global positions
    uint32_t* curY;
    uint64_t yt_cap;
    uint32_t* ICy;            // local f ids
    uint32_t* VSy;            // f values
    uint32_t* err;            // device error flags of the set
    unsigned long long* yt_need;  // keys the layout needs (+1)
    unsigned long long* f_need;   // first-value ids of the set (+1): the by-first-value row pointers scanned
    uint64_t* yoff;           // nrel + 1: first global y id of each relation
    const uint8_t* roles;     // nrel: RelRole bits (CSRs built for the relation)
};

__device__ __forceinline__ DevTable rel_table(unsigned long long* pool, const RelDev& r) {
    return DevTable{pool + r.tab_off, r.tab_cap - 1, r.probe_lim};
}

// The id scans mark the ids before every kTabMark-th slot (tables hold whole
// marks), from which a relation's ids are counted.
constexpr uint32_t kTabMark = 1024;
struct AssignPoolIdDst {
    AssignIdDst d;
    unsigned long long* marks;
    __device__ void operator()(uint64_t i, uint64_t e, uint64_t v) const {
        if ((i & (kTabMark - 1)) == 0) marks[i / kTabMark] = e;
        d(i, e, v);
    }
};

// (Counting the new keys per relation here, with a match over the warp for
// each column, took this pass from 1.3 to 2.4 times the single join's per
// tuple; the id scans have the counts for nothing.)
static __global__ void k_ix_insert(RelPools P) {
    SegCursor sc{P.tup_off, P.nrel};
    DIM3G_FOR_CHUNK(i, P.ntot) {
        const uint32_t r = sc.at(i);
        const uint2 t = P.in[r].pairs[i - sc.lo];
        const uint64_t to = __ldg(&P.tab_off[r]), cap = __ldg(&P.tab_off[r + 1]) - to;
        table_insert(DevTable{P.TF + to, cap - 1, P.probe_lim}, t.x, P.err);
        table_insert(DevTable{P.TY + to, cap - 1, P.probe_lim}, t.y, P.err);
    }
}

// Distinct-key sketches of every relation's two columns (kSketchRegs
// registers per column, zeroed by the caller): relation r's first column at
// regs + 2 r kSketchRegs, its y column after it.  Grid-ordered, so a warp's
// updates fall in one or two relations' registers.
static __global__ void k_rel_sketch(RelPools P, uint32_t* regs) {
    SegCursor sc{P.tup_off, P.nrel};
    DIM3G_FOR_CHUNK(i, P.ntot) {
        const uint32_t r = sc.at(i);
        const uint2 t = P.in[r].pairs[i - sc.lo];
        uint32_t* rr = regs + (uint64_t)2 * r * kSketchRegs;
        sketch_add_if_larger(rr, t.x);
        sketch_add_if_larger(rr + kSketchRegs, t.y);
    }
}

// One warp per column: (sum of 2^-register, zero registers).
static __global__ void k_rel_sketch_sum(const uint32_t* __restrict__ regs, uint32_t ncol, double2* out) {
    const uint32_t col = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x & 31;
    if (col >= ncol) return;
    const uint32_t* r = regs + (uint64_t)col * kSketchRegs;
    double sum = 0;
    uint32_t zeros = 0;
    for (uint32_t k = lane; k < kSketchRegs; k += 32) {
        const uint32_t v = r[k];
        sum += ldexp(1.0, -(int)v);
        zeros += v == 0;
    }
    for (int o = 16; o; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        zeros += __shfl_xor_sync(0xffffffffu, zeros, o);
    }
    if (lane == 0) out[col] = make_double2(sum, (double)zeros);
}

// One CTA: per-relation id bases, z tiling and (y, tile) key ranges.
static __global__ void __launch_bounds__(1024) k_ix_layout(RelPools P, uint32_t tile_lg) {
    __shared__ uint64_t sm[1024 / 32 + 1];
    uint64_t cf = 0, cy = 0, ck = 0;
    for (uint32_t b = 0; b < P.nrel; b += 1024) {
        const uint32_t r = b + threadIdx.x;
        uint64_t nf = 0, ny = 0, T = 1, keys = 0;
        if (r < P.nrel) {
            const uint64_t t0 = P.tab_off[r] / kTabMark, t1 = P.tab_off[r + 1] / kTabMark;
            nf = P.tabF[t1] - P.tabF[t0];
            ny = P.tabY[t1] - P.tabY[t0];
            P.nf_cnt[r] = nf;
            P.ny_cnt[r] = ny;
            T = nf > (1ull << tile_lg) ? (nf + (1ull << tile_lg) - 1) >> tile_lg : 1;
            keys = ny * T + T;  // T sentinel keys: y id ny has no tuples
        }
        uint64_t tf, ty, tk;
        const uint64_t ef = block_excl_scan<1024>(nf, sm, &tf);
        const uint64_t ey = block_excl_scan<1024>(ny, sm, &ty);
        const uint64_t ek = block_excl_scan<1024>(keys, sm, &tk);
        if (r < P.nrel) {
            RelDev d;
            d.nt = P.in[r].n;
            d.tup_off = P.tup_off[r];
            d.tab_off = P.tab_off[r];
            d.tab_cap = P.tab_off[r + 1] - P.tab_off[r];
            d.nf = nf;
            d.ny = ny;
            d.fbase = cf + ef;
            d.ybase = cy + ey;
            d.yt_base = ck + ek;
            d.T = (uint32_t)T;
            d.tile_shift = T > 1 ? tile_lg : 31;
            d.tile_width = T > 1 ? (1u << tile_lg) : (uint32_t)(nf > 0 ? nf : 1);
            d.probe_lim = P.probe_lim;
            P.rel[r] = d;
            P.yoff[r] = d.ybase;
            // a relation without the by-first-value CSR still takes its
            // tuples' positions in that CSR's global prefix (at its first
            // id, in one add), so every relation's positions stay
            // [tup_off, tup_off + nt) for the ones that have it
            if (!(P.roles[r] & kRoleRows) && d.nt) atomicAdd(&P.degF[d.fbase], (uint32_t)d.nt);
        }
        cf += tf;
        cy += ty;
        ck += tk;
    }
    if (threadIdx.x == 0) {
        P.yoff[P.nrel] = cy;
        *P.f_need = cf + 1;
        *P.yt_need = ck + 1;
        if (ck + 1 > P.yt_cap) raise_error(P.err, kErrTableFull);
        // a sketch-sized table overflowed its probe bound: some ids are
        // missing, so no later kernel may use the tables (the host rebuilds
        // with tuple-sized tables)
        if (*(volatile uint32_t*)P.err & kErrProbeLimit) *P.yt_need = ~0ull;
    }
}

// Tuples -> (global f id, global y id); degree of f; count of (y, f tile).
static __global__ void k_ix_map(RelPools P) {
    if (*P.yt_need > P.yt_cap) return;  // layout overflow: the host regrows
    SegCursor sc{P.tup_off, P.nrel};
    DIM3G_FOR_CHUNK(i, P.ntot) {
        const uint32_t r = sc.at(i);
        const RelDev& d = P.rel[r];
        const uint2 t = P.in[r].pairs[i - sc.lo];
        const uint32_t fid = table_find(rel_table(P.TF, d), t.x);
        const uint32_t yid = table_find(rel_table(P.TY, d), t.y);
        P.Pm[i] = make_uint2(fid, yid);
        const uint8_t ro = P.roles[r];
        if (ro & kRoleRows) atomicAdd(&P.degF[fid], 1u);
        if (ro & kRoleCols) {
            const uint64_t key = d.yt_base + (uint64_t)(yid - d.ybase) * d.T + ((fid - d.fbase) >> d.tile_shift);
            atomic_inc_agg(P.cnt_yt, key);  // heavy y keys repeat within a warp
        }
    }
}

static __global__ void k_ix_scatter(RelPools P) {
    if (*P.yt_need > P.yt_cap) return;
    SegCursor sc{P.tup_off, P.nrel};
    DIM3G_FOR_CHUNK(i, P.ntot) {
        const uint32_t r = sc.at(i);
        const RelDev& d = P.rel[r];
        const uint2 pm = P.Pm[i];
        const uint8_t ro = P.roles[r];
        const uint32_t fl = pm.x - (uint32_t)d.fbase;
        if (ro & kRoleRows) {
            const uint32_t pos = atomicAdd(&P.curF[pm.x], 1u);
            P.ICf[pos] = pm.y;
        }
        if (ro & kRoleCols) {
            const uint64_t key = d.yt_base + (uint64_t)(pm.y - d.ybase) * d.T + (fl >> d.tile_shift);
            const uint32_t p2 = atomic_inc_agg(P.curY, key);
            P.ICy[p2] = fl;
            P.VSy[p2] = P.in[r].pairs[i - sc.lo].x;
        }
    }
}

// Exact join size of every ordered relation pair (r, s):
// outj[r * nrel + s] = sum over y of deg_r(y) * deg_s(y).  One thread per y
// of the set (global y ids), probing every relation's y table.
static __global__ void k_pair_outj(RelPools P, unsigned long long* outj) {
    if (*P.yt_need > P.yt_cap) return;
    const uint64_t ny_all = P.yoff[P.nrel];
    SegCursor sc{P.yoff, P.nrel};
    DIM3G_FOR_CHUNK(g, ny_all) {
        const uint32_t r = sc.at(g);
        const RelDev& d = P.rel[r];
        const uint32_t* jr = P.JRy + d.yt_base + (g - sc.lo) * d.T;
        const unsigned long long deg_r = jr[d.T] - jr[0];
        const uint32_t v = P.id2y[g];
        for (uint32_t s = 0; s < P.nrel; s++) {
            const RelDev& e = P.rel[s];
            const uint32_t t = table_find(rel_table(P.TY, e), v);
            if (t == kNotFound) continue;
            const uint32_t* js = P.JRy + e.yt_base + (uint64_t)(t - e.ybase) * e.T;
            const uint64_t key = (uint64_t)r * P.nrel + s;
            atomic_add_grouped(&outj[key], key, deg_r * (js[e.T] - js[0]));
        }
    }
}

// --------------------------------------------------------------- query set
enum QueryOp : uint32_t { kOpProject = 0, kOpCount = 1 };

struct QueryIn {
    uint32_t p, q;        // relation ids: P drives the rows, Q is probed
    uint32_t op;          // QueryOp
    uint32_t pad;
    uint2* out;           // (P.f, Q.f) pairs
    unsigned long long* out_cnt;  // counts (kOpCount)
    uint64_t cap;         // pairs the output holds
};

// Per-query results, copied back after the batch.
struct QueryRes {
    unsigned long long n_out;   // pairs written (or needed when > cap)
    unsigned long long out_j;   // candidates
    uint32_t err;
    uint32_t nx, ny, nz;        // rows (distinct P.f; 0 when a side is empty), P.y, Q.f
};

constexpr uint32_t kCountBuckets = 8, kNoBucket = 0xFF;
// A row of more than kQLongRow entries, past the first that its lanes take, is
// worked out in pieces of kQPiece by the whole grid (k_q_long).
constexpr uint32_t kQLongRow = 4096, kQPiece = 2048;
struct QLongRow {
    unsigned long long w;  // candidates so far
    uint64_t g;            // row of the row space
    uint32_t qi, e1;
    uint32_t left;         // pieces not done
};
// Rows and pieces that n entries may have.
inline uint64_t q_long_rows(uint64_t n) { return n / kQLongRow + 1; }
inline uint64_t q_pieces(uint64_t n) { return n / kQPiece + n / kQLongRow + 1; }

struct QueryPools {
    const RelDev* rel;
    const QueryIn* qin;
    uint32_t nq;
    const uint64_t* qt_off;    // nq + 1: prefix of P tuple counts (y map, P entries)
    const uint64_t* qrow_off;  // nq + 1: prefix of P tuple counts + 1 (rows)
    uint64_t ntot, nrows;
    const unsigned long long* TY;
    const uint32_t* id2f;
    const uint32_t* id2y;
    const uint32_t* JRf;
    const uint32_t* ICf;
    const uint32_t* JRy;
    const uint32_t* ICy;
    const uint32_t* VSy;
    uint2* ymap;      // ntot: per y id of P, Q's y id and its tuples
    uint64_t* step_off;  // nq + 1: prefix of the queries' warp steps (k_q_work)
    uint32_t* ICq;    // ntot: P entries as Q y ids
    uint32_t* JRq;    // nrows: P row pointers, relative
    uint32_t* ucap;   // nrows
    uint8_t* bucket;  // nrows: RowBuckets, COUNT rows from kCountBuckets on
    unsigned long long* nbucket[2];  // rows per bucket: join-project, COUNT
    QLongRow* longs;
    uint2* pieces;    // of the long rows: slot in longs, first entry
    unsigned long long* n_long;  // long rows, and their pieces
    RowCtx* rc;       // nq
    Reserve* rs;      // nq
    QueryRes* res;    // nq
    const unsigned long long* yt_need;  // the relation set's key-space check
    uint64_t yt_cap;
    uint32_t cta_rr;  // the context's CTA-row walk (RowCtx::cta_rr)
};

// False when the relation set's (y, f tile) key space outgrew its pool: its
// CSR was not built, and the query kernels must not read it.
__device__ __forceinline__ bool layout_ok(const QueryPools& Q) { return *Q.yt_need <= Q.yt_cap; }

// y map: y id of P -> y id of Q, or Q's sentinel y id (no tuples).
static __global__ void k_q_ymap(QueryPools Q) {
    if (!layout_ok(Q)) return;
    SegCursor sc{Q.qt_off, Q.nq};
    DIM3G_FOR_CHUNK(i, Q.ntot) {
        const uint32_t qi = sc.at(i);
        const QueryIn qn = Q.qin[qi];
        const RelDev& p = Q.rel[qn.p];
        const RelDev& q = Q.rel[qn.q];
        const uint64_t y = i - sc.lo;
        if (y >= p.ny) continue;
        const uint32_t g = table_find(rel_table((unsigned long long*)Q.TY, q), Q.id2y[p.ybase + y]);
        const uint32_t yq = g == kNotFound ? (uint32_t)q.ny : g - (uint32_t)q.ybase;
        const uint32_t* jr = Q.JRy + q.yt_base + (uint64_t)yq * q.T;
        Q.ymap[i] = make_uint2(yq, jr[q.T] - jr[0]);
    }
}

// Lanes a row (log2) of a query's k_q_work steps (as row_work_lanes).
__device__ __forceinline__ uint32_t query_lanes(const RelDev& p) {
    const uint64_t per_row = p.nf ? p.nt / p.nf : 0;
    return per_row > 64 ? 5u : (per_row > 24 ? 4u : (per_row > 8 ? 3u : 2u));
}

// A query's row context and output reservation.
__device__ __forceinline__ void query_setup(const QueryPools& Q, uint32_t qi) {
    const QueryIn qn = Q.qin[qi];
    const RelDev& p = Q.rel[qn.p];
    const RelDev& q = Q.rel[qn.q];
    RowCtx c{};
    c.JR_R = Q.JRq + Q.qrow_off[qi];
    c.IC_R = Q.ICq + Q.qt_off[qi];
    c.JR_S = Q.JRy + q.yt_base;
    c.IC_S = Q.ICy;
    c.VS = Q.VSy;
    c.T = q.T;
    c.tile_width = q.tile_width;
    c.m = (uint32_t)q.nf;
    c.cta_rr = Q.cta_rr;
    c.ucap = Q.ucap + Q.qrow_off[qi];
    c.cnt = nullptr;
    c.off = nullptr;
    c.id2x = Q.id2f + p.fbase;
    c.id2z = Q.id2f + q.fbase;
    c.out = qn.out;
    c.err = &Q.res[qi].err;
    c.next_row = nullptr;
    Q.rc[qi] = c;
    Q.rs[qi] = Reserve{&Q.res[qi].n_out, qn.cap};
    QueryRes r{};
    const bool ok = layout_ok(Q);
    const bool live = ok && Q.qt_off[qi + 1] > Q.qt_off[qi];  // both sides nonempty
    r.nx = live ? (uint32_t)p.nf : 0u;
    r.err = ok ? 0u : (uint32_t)kErrTableFull;
    r.ny = (uint32_t)p.ny;
    r.nz = (uint32_t)q.nf;
    Q.res[qi] = r;
}

// One CTA: every query's setup, and the warp steps of its rows (the rows of a
// step share a warp; nx + 1 row pointers).
static __global__ void __launch_bounds__(1024) k_q_setup(QueryPools Q) {
    __shared__ uint64_t sm[1024 / 32 + 1];
    uint64_t carry = 0;
    for (uint32_t b = 0; b < Q.nq; b += 1024) {
        const uint32_t qi = b + threadIdx.x;
        uint64_t steps = 0;
        if (qi < Q.nq) {
            query_setup(Q, qi);
            const uint32_t per = 32u >> query_lanes(Q.rel[Q.qin[qi].p]);
            steps = layout_ok(Q) ? (Q.res[qi].nx + per) / per : 0;
        }
        uint64_t sum;
        const uint64_t e = block_excl_scan<1024>(steps, sm, &sum);
        if (qi < Q.nq) Q.step_off[qi] = carry + e;
        carry += sum;
    }
    if (threadIdx.x == 0) Q.step_off[Q.nq] = carry;
}

// A row with its candidates counted: its distinct bound and bucket (kRowBuckets:
// none).
__device__ __forceinline__ uint32_t query_row(const QueryPools& Q, const RowBuckets& rb, uint32_t qi, uint64_t g,
                                              uint32_t ne, unsigned long long w, uint32_t m, uint32_t fam) {
    const uint32_t u = (uint32_t)(w < m ? w : m);
    const uint32_t k = rb.of(row_class(w, u, ne, rb.cap_w, fam ? agg_cap_b(m, rb.cap_b) : rb.cap_b, rb.tiny), u);
    Q.ucap[g] = u;
    if (fam && w >= 0xFFFFFFFFull) raise_error(&Q.res[qi].err, kErrCountRange);
    if (k < kRowBuckets) Q.bucket[g] = (uint8_t)(fam * kCountBuckets + k);
    return k;
}

// The rows of all queries: P's entries as Q's y ids, P's row pointers, the
// row's candidates and its bucket.  A warp step is 32 >> lg rows of one query,
// 2^lg lanes a row, about as many as its rows have entries on average (a row
// of more than 4 x 2^lg is finished by the whole warp; see k_row_work).  Row
// space planned from tuple counts, past a query's distinct first values, is
// not visited.  An entry costs one random sector (its y id's ymap pair).
// Rows of more than kQLongRow entries are left to k_q_long: a hub of 2M entries
// among 4M held one warp for 28.7 ms.
// In place of three passes with a per-entry atomic on the row's candidates
// (16 resident queries of 35M entries: 1020 us; 48-join batch: 345 us).
static __global__ void __launch_bounds__(256) k_q_work(QueryPools Q, RowBuckets rb) {
    __shared__ uint32_t s_n[2][kRowBuckets + 1];
    if (threadIdx.x < 2 * (kRowBuckets + 1)) s_n[threadIdx.x / (kRowBuckets + 1)][threadIdx.x % (kRowBuckets + 1)] = 0;
    __syncthreads();
    const uint32_t lane = lane_id();
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint64_t steps = layout_ok(Q) ? Q.step_off[Q.nq] : 0;
    uint64_t lo = 1, hi = 0;  // steps of the warp's query
    uint32_t qi = 0, nx = 0, m = 0, fam = 0, lg = 5, tup_off = 0;
    const uint32_t* jp = nullptr;  // P's row pointers (from tup_off on)
    const uint32_t* icf = nullptr;  // P's entries (global y ids)
    const uint2* ymap = nullptr;    // indexed by P's global y id
    uint32_t* icq = nullptr;
    unsigned long long acc = 0;  // candidates of the warp's query, lane's share
    for (uint64_t s = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < steps; s += nwarps) {
        if (s < lo || s >= hi) {
            acc = warp_sum(acc);
            if (lane == 0 && acc) atomicAdd(&Q.res[qi].out_j, acc);
            acc = 0;
            qi = seg_find(Q.step_off, Q.nq, s);
            lo = Q.step_off[qi];
            hi = Q.step_off[qi + 1];
            const QueryIn qn = Q.qin[qi];
            const RelDev& p = Q.rel[qn.p];
            nx = Q.res[qi].nx;
            m = Q.res[qi].nz;
            fam = qn.op == kOpCount;
            lg = query_lanes(p);
            tup_off = (uint32_t)p.tup_off;
            jp = Q.JRf + p.fbase;
            icf = Q.ICf + p.tup_off;
            ymap = Q.ymap + Q.qt_off[qi] - p.ybase;
            icq = Q.ICq + Q.qt_off[qi];
        }
        const uint32_t G = 1u << lg, gl = lane & (G - 1);
        const uint64_t x = ((s - lo) << (5 - lg)) + (lane >> lg), g = Q.qrow_off[qi] + x;
        const bool live = x < nx;
        uint32_t e0 = 0, e1 = 0;
        if (x <= nx) {
            e0 = jp[x] - tup_off;
            if (gl == 0) Q.JRq[g] = e0;
            e1 = live ? jp[x + 1] - tup_off : e0;
        }
        unsigned long long w = 0;
        const uint32_t head = e0 + min(e1 - e0, 4 * G);
        uint32_t y[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) y[k] = e0 + gl + k * G < head ? __ldg(&icf[e0 + gl + k * G]) : kEmpty32;
#pragma unroll
        for (uint32_t k = 0; k < 4; k++)
            if (y[k] != kEmpty32) {
                const uint2 t = __ldg(&ymap[y[k]]);
                icq[e0 + gl + k * G] = t.x;
                w += t.y;
            }
        // the rest of the warp's long rows, all lanes on one row at a time, or
        // its pieces for k_q_long
        uint32_t slot = kEmpty32;
        for (uint32_t longs = __ballot_sync(0xffffffffu, gl == 0 && head < e1); longs; longs &= longs - 1) {
            const int src = __ffs(longs) - 1;
            const uint32_t b0 = __shfl_sync(0xffffffffu, head, src), b1 = __shfl_sync(0xffffffffu, e1, src);
            if (b1 - b0 > kQLongRow) {
                const uint32_t np = (b1 - b0 - 1) / kQPiece + 1;
                uint32_t sl = 0;
                unsigned long long at = 0;
                if (lane == 0) {
                    sl = (uint32_t)atomicAdd(&Q.n_long[0], 1ull);
                    at = atomicAdd(&Q.n_long[1], (unsigned long long)np);
                }
                sl = __shfl_sync(0xffffffffu, sl, 0);
                at = __shfl_sync(0xffffffffu, at, 0);
                if ((int)lane == src) {
                    slot = sl;
                    Q.longs[sl] = QLongRow{0, g, qi, b1, np};
                }
                for (uint32_t k = lane; k < np; k += 32) Q.pieces[at + k] = make_uint2(sl, b0 + k * kQPiece);
                continue;
            }
            unsigned long long v = 0;
#pragma unroll 4
            for (uint32_t e = b0 + lane; e < b1; e += 32) {
                const uint2 t = __ldg(&ymap[__ldg(&icf[e])]);
                icq[e] = t.x;
                v += t.y;
            }
            v = warp_sum(v);
            if ((int)lane == src) w += v;
        }
        for (uint32_t o = G >> 1; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
        if (gl == 0 && live) {
            if (slot == kEmpty32) {
                const uint32_t k = query_row(Q, rb, qi, g, e1 - e0, w, m, fam);
                acc += w;
                if (k < kRowBuckets) atomicAdd(&s_n[fam][k], 1u);
            } else {
                Q.longs[slot].w = w;
            }
        }
    }
    acc = warp_sum(acc);
    if (lane == 0 && acc) atomicAdd(&Q.res[qi].out_j, acc);
    __syncthreads();
    if (threadIdx.x < 2 * (kRowBuckets + 1)) {
        const uint32_t fam = threadIdx.x / (kRowBuckets + 1), k = threadIdx.x % (kRowBuckets + 1);
        if (k < kRowBuckets && s_n[fam][k]) atomicAdd(&Q.nbucket[fam][k], (unsigned long long)s_n[fam][k]);
    }
}

// The long rows that k_q_work left, a warp a piece; whoever does a row's last
// piece bins it.
static __global__ void __launch_bounds__(256) k_q_long(QueryPools Q, RowBuckets rb) {
    const uint32_t lane = lane_id();
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5, n = Q.n_long[1];
    for (uint64_t t = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < n; t += nwarps) {
        const uint2 piece = Q.pieces[t];
        QLongRow& l = Q.longs[piece.x];
        const uint32_t qi = l.qi, b0 = piece.y, ne = min(l.e1 - b0, kQPiece);
        const QueryIn qn = Q.qin[qi];
        const RelDev& p = Q.rel[qn.p];
        const uint32_t* icf = Q.ICf + p.tup_off + b0;
        const uint2* ymap = Q.ymap + Q.qt_off[qi] - p.ybase;
        uint32_t* icq = Q.ICq + Q.qt_off[qi] + b0;
        unsigned long long v = 0;
#pragma unroll 4
        for (uint32_t e = lane; e < ne; e += 32) {
            const uint2 y = __ldg(&ymap[__ldg(&icf[e])]);
            icq[e] = y.x;
            v += y.y;
        }
        v = warp_sum(v);
        if (lane == 0) {
            if (v) atomicAdd(&l.w, v);
            __threadfence();
            if (atomicSub(&l.left, 1u) == 1u) {
                __threadfence();
                const unsigned long long w = atomicAdd(&l.w, 0ull);
                const uint32_t fam = qn.op == kOpCount, k = query_row(Q, rb, qi, l.g, kQLongRow, w, Q.res[qi].nz, fam);
                if (w) atomicAdd(&Q.res[qi].out_j, w);
                if (k < kRowBuckets) atomicAdd(&Q.nbucket[fam][k], 1ull);
            }
        }
        __syncwarp();
    }
}

// Row g of the row space -> (query, local row).
__device__ __forceinline__ uint32_t query_of_row(const QueryPools& Q, uint32_t g, uint32_t* x) {
    const uint32_t qi = seg_find(Q.qrow_off, Q.nq, g);
    *x = g - (uint32_t)Q.qrow_off[qi];
    return qi;
}

struct BatchRows {
    const uint32_t* list;
    const unsigned long long* n_a;  // rows of the list (or its first part)
    const unsigned long long* n_b;  // second part (or nullptr)
    uint32_t* next;                 // dynamic row counter of CTA classes
    const unsigned long long* skip0 = nullptr;  // the rows start past these counts (device; null: 0)
    const unsigned long long* skip1 = nullptr;
    __device__ __forceinline__ const uint32_t* rows() const {
        return list + (skip0 ? *skip0 : 0ull) + (skip1 ? *skip1 : 0ull);
    }
};

// ---- project, single pass: rows of many queries, each CTA (or warp) copying
// its row's query context into shared memory; the row bodies of single.cuh.
static __global__ void __launch_bounds__(1024) k_b_single_bitmap(QueryPools Q, BatchRows L, uint32_t bitmap_words) {
    extern __shared__ uint32_t bm[];
    __shared__ uint32_t s_row, s_x, s_q;
    __shared__ RowCtx s_c;
    __shared__ CtaChunks s_cc;
    if (threadIdx.x == 0) s_cc.n = 0;
    uint32_t* stage = bm + bitmap_words + (threadIdx.x >> 5) * kStage;
    const uint32_t nrows = (uint32_t)(*L.n_a + *L.n_b);
    for (uint32_t ri = cta_next_row(L.next, &s_row); ri < nrows; ri = cta_next_row(L.next, &s_row)) {
        if (threadIdx.x == 0) {
            uint32_t x;
            s_q = query_of_row(Q, L.list[ri], &x);
            s_x = x;
            s_c = Q.rc[s_q];
        }
        __syncthreads();
        StageSink sink{stage, s_c.out, Q.rs[s_q], s_c.id2x[s_x]};
        single_bitmap_row(s_c, s_x, bm, sink, &s_cc);
        sink.flush();
    }
}

static __global__ void __launch_bounds__(1024) k_b_single_block(QueryPools Q, BatchRows L, uint32_t block_lg) {
    extern __shared__ uint32_t smem[];
    __shared__ uint32_t s_row, s_x, s_q;
    __shared__ RowCtx s_c;
    __shared__ CtaChunks s_cc;
    if (threadIdx.x == 0) s_cc.n = 0;
    uint32_t* stage = smem + (1u << block_lg) + (threadIdx.x >> 5) * kStage;
    const uint32_t nrows = (uint32_t)*L.n_a;
    const uint32_t* rows = L.rows();
    for (uint32_t ri = cta_next_row(L.next, &s_row); ri < nrows; ri = cta_next_row(L.next, &s_row)) {
        if (threadIdx.x == 0) {
            uint32_t x;
            s_q = query_of_row(Q, rows[ri], &x);
            s_x = x;
            s_c = Q.rc[s_q];
        }
        __syncthreads();
        StageSink sink{stage, s_c.out, Q.rs[s_q], s_c.id2x[s_x]};
        single_block_row(s_c, s_x, smem, sink, block_lg, &s_cc);
        sink.flush();
    }
}

// Warp class: at most 8 warps per CTA, one context slot each.
static __global__ void __launch_bounds__(256) k_b_single_warp(QueryPools Q, BatchRows L, uint32_t warp_lg,
                                                              uint32_t stage) {
    extern __shared__ uint32_t smem[];
    __shared__ RowCtx s_c[8];
    const uint32_t nw = blockDim.x >> 5, wib = threadIdx.x >> 5, lane = lane_id();
    uint32_t* tab = smem + (size_t)wib * warp_row_words(warp_lg, stage);
    // the warp's pairs are staged across its rows and flushed when the
    // query (cursor and output) changes
    PairStageSink sink{reinterpret_cast<uint2*>(tab + (1u << warp_lg)), nullptr, Reserve{nullptr, 0}, 0, stage};
    uint32_t cur_q = 0xFFFFFFFFu, q_lo = 1, q_hi = 0;
    const uint32_t nrows = (uint32_t)*L.n_a;
    for (uint32_t ri = blockIdx.x * nw + wib; ri < nrows; ri += gridDim.x * nw) {
        // rows of one query are contiguous in the list: look the query up
        // only when the row leaves the current query's row range
        const uint32_t g = L.list[ri];
        uint32_t qi = cur_q;
        if (g < q_lo || g >= q_hi) {
            qi = seg_find(Q.qrow_off, Q.nq, g);
            q_lo = (uint32_t)Q.qrow_off[qi];
            q_hi = (uint32_t)Q.qrow_off[qi + 1];
        }
        const uint32_t x = g - q_lo;
        if (qi != cur_q) {
            sink.flush();
            __syncwarp();
            if (lane == 0) s_c[wib] = Q.rc[qi];
            __syncwarp();
            sink.rs = Q.rs[qi];
            sink.out = s_c[wib].out;
            cur_q = qi;
        }
        single_warp_row(s_c[wib], x, tab, sink, warp_lg);
    }
    sink.flush();
}

// The query of the pack list's row in lane `lo` (g: the lanes' rows), tried
// against the warp's current query first.
__device__ __forceinline__ uint32_t pack_query_of(const QueryPools& Q, uint32_t g, uint32_t lo, uint32_t cur_q) {
    const uint32_t g0 = __shfl_sync(0xffffffffu, g, lo);
    if (cur_q != 0xFFFFFFFFu && g0 >= (uint32_t)Q.qrow_off[cur_q] && g0 < (uint32_t)Q.qrow_off[cur_q + 1]) return cur_q;
    return seg_find(Q.qrow_off, Q.nq, g0);
}
// The end of the run of lanes [lo, end) whose rows belong to query qi, whose
// rows start at *q_lo.
__device__ __forceinline__ uint32_t pack_query_end(const QueryPools& Q, uint32_t g, uint32_t lo, uint32_t n, uint32_t qi,
                                                   uint32_t* q_lo) {
    *q_lo = (uint32_t)Q.qrow_off[qi];
    const uint32_t q_hi = (uint32_t)Q.qrow_off[qi + 1], lane = lane_id();
    const uint32_t other = __ballot_sync(0xffffffffu, lane >= lo && lane < n && (g < *q_lo || g >= q_hi));
    return other ? __ffs(other) - 1 : n;
}

// Tiny rows: packs of rows of one query (packed.cuh), at most 8 warps a CTA
// with a context slot each.  A pack ends where the list goes on to another
// query.
static __global__ void __launch_bounds__(256, 4) k_b_single_pack(QueryPools Q, BatchRows L) {
    extern __shared__ uint32_t smem[];
    __shared__ RowCtx s_c[8];
    const uint32_t nw = blockDim.x >> 5, wib = threadIdx.x >> 5, lane = lane_id();
    uint32_t* tab = smem + (size_t)wib * kPackWords;
    PackSink sink{reinterpret_cast<uint2*>(tab + (1u << kPackLg)), nullptr, Reserve{nullptr, 0}};
    uint32_t cur_q = 0xFFFFFFFFu;
    const uint32_t nrows = (uint32_t)*L.n_a, warps = gridDim.x * nw;
    uint32_t take = (nrows + warps - 1) / warps;
    take = take > 32 ? 32 : take;
    for (uint64_t r0 = (uint64_t)(blockIdx.x * nw + wib) * take; r0 < nrows; r0 += (uint64_t)warps * take) {
        const uint32_t n = (uint32_t)min((uint64_t)take, nrows - r0);
        const uint32_t g = lane < n ? L.list[r0 + lane] : 0xFFFFFFFFu;
        for (uint32_t lo = 0; lo < n;) {
            const uint32_t qi = pack_query_of(Q, g, lo, cur_q);
            uint32_t q_lo;
            const uint32_t hi = pack_query_end(Q, g, lo, n, qi, &q_lo);
            if (qi != cur_q) {
                sink.flush();
                __syncwarp();
                if (lane == 0) s_c[wib] = Q.rc[qi];
                __syncwarp();
                sink.rs = Q.rs[qi];
                sink.out = s_c[wib].out;
                cur_q = qi;
            }
            pack_rows(s_c[wib], lane >= lo && lane < hi ? g - q_lo : 0u, lo, hi, tab, sink);
            lo = hi;
        }
    }
    sink.flush();
}

// ---- COUNT, single pass: the row forms of aggregate.cuh, groups to each
// query's cursor.
__device__ __forceinline__ AggOut query_agg(const QueryPools& Q, uint32_t qi) {
    return AggOut{Q.qin[qi].out_cnt, SumAcc{}, Q.rs[qi]};
}

static __global__ void __launch_bounds__(256, 4) k_b_agg_pack(QueryPools Q, BatchRows L) {
    extern __shared__ uint32_t smem[];
    __shared__ RowCtx s_c[8];
    const uint32_t nw = blockDim.x >> 5, wib = threadIdx.x >> 5, lane = lane_id();
    uint32_t* keys = smem + (size_t)wib * kAggPackWords;
    uint32_t* stage = keys + (2u << kAggPackLg);
    GroupStage gs{reinterpret_cast<uint2*>(stage), stage + 2 * kAggPackStage, nullptr, nullptr, Reserve{nullptr, 0},
                  kAggPackStage};
    uint32_t cur_q = 0xFFFFFFFFu;
    const uint32_t nrows = (uint32_t)*L.n_a, warps = gridDim.x * nw;
    uint32_t take = (nrows + warps - 1) / warps;
    take = take > 32 ? 32 : take;
    for (uint64_t r0 = (uint64_t)(blockIdx.x * nw + wib) * take; r0 < nrows; r0 += (uint64_t)warps * take) {
        const uint32_t n = (uint32_t)min((uint64_t)take, nrows - r0);
        const uint32_t g = lane < n ? L.list[r0 + lane] : 0xFFFFFFFFu;
        for (uint32_t lo = 0; lo < n;) {
            const uint32_t qi = pack_query_of(Q, g, lo, cur_q);
            uint32_t q_lo;
            const uint32_t hi = pack_query_end(Q, g, lo, n, qi, &q_lo);
            if (qi != cur_q) {
                gs.flush();
                __syncwarp();
                if (lane == 0) s_c[wib] = Q.rc[qi];
                __syncwarp();
                const AggOut ao = query_agg(Q, qi);
                gs.rs = ao.rs;
                gs.out = s_c[wib].out;
                gs.out_cnt = ao.cnt;
                cur_q = qi;
            }
            agg_pack_rows(s_c[wib], lane >= lo && lane < hi ? g - q_lo : 0u, lo, hi, keys, gs);
            lo = hi;
        }
    }
    gs.flush();
}

static __global__ void __launch_bounds__(1024, 1) k_b_agg_map(QueryPools Q, BatchRows L, uint32_t lg) {
    extern __shared__ uint32_t smem[];
    __shared__ uint32_t s_row, s_x, s_q, s_pos;
    __shared__ RowCtx s_c;
    __shared__ CtaChunks s_cc;
    const uint32_t nrows = (uint32_t)*L.n_a;
    const uint32_t* rows = L.rows();
    for (uint32_t ri = cta_next_row(L.next, &s_row); ri < nrows; ri = cta_next_row(L.next, &s_row)) {
        if (threadIdx.x == 0) {
            uint32_t x;
            s_q = query_of_row(Q, rows[ri], &x);
            s_x = x;
            s_c = Q.rc[s_q];
        }
        __syncthreads();
        agg_map_row(s_c, query_agg(Q, s_q), s_x, smem, lg, &s_cc, &s_pos);
    }
}

// Ranked rows: a row's z tiles are taken in turn; the next row is claimed, and
// its query and header looked up, during the current one.
static __global__ void __launch_bounds__(1024, 1) k_b_agg_ranked(QueryPools Q, BatchRows L, size_t smem_bytes,
                                                                uint32_t* ctr, uint32_t tile_lg) {
    extern __shared__ uint32_t smem[];
    __shared__ uint32_t s_q[2], s_pos, s_wbase[33];
    __shared__ unsigned long long s_base;
    __shared__ RankHead s_head[2];
    __shared__ RowCtx s_c[2];
    __shared__ CtaChunks s_cc;
    const uint32_t nrows = (uint32_t)(*L.n_a + *L.n_b);
    auto claim = [&](uint32_t k) {
        const uint32_t i = atomicAdd(L.next, 1u);
        s_head[k].item = i;
        if (i >= nrows) return;
        uint32_t x;
        s_q[k] = query_of_row(Q, L.list[i], &x);
        s_c[k] = Q.rc[s_q[k]];
        s_head[k] = rank_head(s_c[k], i, x, 0);
    };
    if (threadIdx.x == 0) claim(0);
    __syncthreads();
    for (uint32_t k = 0; s_head[k].item < nrows; k ^= 1) {
        const RowCtx& c = s_c[k];
        const AggOut ao = query_agg(Q, s_q[k]);
        const RankHead h = s_head[k];
        const RankLayout l = rank_layout(c.tile_width, blockDim.x >> 5, smem_bytes);
        for (uint32_t t = 0; t < c.T; t++) {
            agg_ranked_tile(c, ao, h, t, smem, l, &s_cc, &s_pos, s_wbase, &s_base, ctr + ((size_t)blockIdx.x << tile_lg), [&] {
                if (t == 0) claim(k ^ 1);
            });
            __syncthreads();
        }
    }
}

}  // namespace dim3g
