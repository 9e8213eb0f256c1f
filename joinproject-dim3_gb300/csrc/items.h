// items.h -- index arithmetic of the row kernels near 2^32, free of device
// code, so that the tests run it on the CPU at sizes no device test reaches.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define DIM3G_HD __host__ __device__ __forceinline__
#else
#define DIM3G_HD inline
#endif

namespace dim3g {

// `total` candidates taken `piece` at a time: warps draw piece numbers from a
// shared counter.  (A counter of candidates wraps where total is near 2^32:
// the draws past the end come out at the start again.)
struct Pieces {
    uint32_t piece, total, n;  // n: number of pieces
    DIM3G_HD Pieces(uint32_t piece, uint32_t total) : piece(piece), total(total), n(total / piece + (total % piece != 0)) {}
    // [*p0, *p1) of piece k, or false past the end
    DIM3G_HD bool at(uint32_t k, uint32_t* p0, uint32_t* p1) const {
        if (k >= n) return false;
        *p0 = k * piece;
        *p1 = k + 1 < n ? *p0 + piece : total;
        return true;
    }
};

// Part k < parts of `total` candidates in equal shares; false where it is
// empty.
DIM3G_HD bool share_of(uint32_t k, uint32_t parts, uint32_t total, uint32_t* p0, uint32_t* p1) {
    const uint32_t share = total / parts + (total % parts != 0);
    *p0 = k * share;  // below 2^32: at most total, or less than parts^2
    if (*p0 >= total) return false;
    *p1 = *p0 + (share < total - *p0 ? share : total - *p0);
    return true;
}

// Work items of rows taken `per` z tiles apart: item i is tile i % per of row
// i / per.  33M heavy rows over 128 tiles are 2^32 of them.
struct TileItems {
    uint64_t rows;
    uint32_t per;
    DIM3G_HD uint64_t count() const { return rows * per; }
    DIM3G_HD uint32_t row(uint64_t i) const { return (uint32_t)(i / per); }
    DIM3G_HD uint32_t tile(uint64_t i) const { return (uint32_t)(i % per); }
};

}  // namespace dim3g
