"""The row kernels' index arithmetic near 2^32 (csrc/items.h), compiled for the
CPU: sizes that would take a device minutes, or never end there, if the
arithmetic wrapped."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "joinproject-dim3_gb300", "csrc")

SRC = r"""
#include "items.h"
using namespace dim3g;
extern "C" {
// Draws pieces 0, 1, ... as `warps` warps do until each has been told that
// there is none left: candidates covered (all ones on a gap, an overlap or
// more draws than pieces and warps), number of pieces in *n.
uint64_t walk(uint32_t piece, uint32_t total, uint32_t warps, uint64_t* n) {
    uint64_t covered = 0;
    uint32_t k = 0, done = 0;
    const Pieces pieces(piece, total);
    *n = 0;
    while (done < warps) {
        uint32_t p0, p1;
        if (!pieces.at(k++, &p0, &p1)) {
            done++;
            continue;
        }
        if (done || p0 != covered || p1 <= p0 || p1 - p0 > piece || p1 > total) return ~0ull;
        covered += p1 - p0;
        ++*n;
    }
    return covered;
}
// The candidates that `parts` equal shares cover, or all ones.
uint64_t shares(uint32_t parts, uint32_t total) {
    uint64_t covered = 0;
    for (uint32_t k = 0; k < parts; k++) {
        uint32_t p0, p1;
        if (!share_of(k, parts, total, &p0, &p1)) continue;
        if (p0 != covered || p1 <= p0 || p1 > total) return ~0ull;
        covered += p1 - p0;
    }
    return covered;
}
uint64_t items(uint64_t rows, uint32_t per) { return TileItems{rows, per}.count(); }
uint32_t item_row(uint64_t rows, uint32_t per, uint64_t i) { return TileItems{rows, per}.row(i); }
uint32_t item_tile(uint64_t rows, uint32_t per, uint64_t i) { return TileItems{rows, per}.tile(i); }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("items")
    src, so = str(d / "items.cpp"), str(d / "items.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", CSRC, src, "-o", so], check=True)
    L = ctypes.CDLL(so)
    L.walk.restype = ctypes.c_uint64
    L.walk.argtypes = [ctypes.c_uint32] * 3 + [ctypes.POINTER(ctypes.c_uint64)]
    L.shares.restype = ctypes.c_uint64
    L.shares.argtypes = [ctypes.c_uint32] * 2
    L.items.restype = ctypes.c_uint64
    L.items.argtypes = [ctypes.c_uint64, ctypes.c_uint32]
    for f in (L.item_row, L.item_tile):
        f.restype = ctypes.c_uint32
        f.argtypes = [ctypes.c_uint64, ctypes.c_uint32, ctypes.c_uint64]
    return L


@pytest.mark.parametrize("piece", [128, 256, 1152, 4096, 1 << 27, (1 << 32) - 1])
@pytest.mark.parametrize("total", [0, 1, 255, 256, 257, 1 << 20, (1 << 32) - 135_168, (1 << 32) - 4097, (1 << 32) - 4096,
                                   (1 << 32) - 1024, (1 << 32) - 256, (1 << 32) - 2, (1 << 32) - 1])
def test_pieces_cover_all_candidates_once(lib, piece, total):
    n = ctypes.c_uint64()
    assert lib.walk(piece, total, 32, ctypes.byref(n)) == total
    assert n.value == -(-total // piece)


@pytest.mark.parametrize("parts", [1, 4, 8, 15, 16, 32])
def test_shares_cover_all_candidates_once(lib, parts):
    for total in [*range(0, 1100), *range((1 << 32) - 1100, 1 << 32)]:
        assert lib.shares(parts, total) == total


@pytest.mark.parametrize("rows,per", [(1, 1), (7, 3), (2_100_000, 2048), (33 << 20, 128), ((1 << 31) - 1, 8192)])
def test_items_of_rows_and_tiles(lib, rows, per):
    """2.1M ranked rows over 2048 tiles, 33M over 128: every row and tile once."""
    n = lib.items(rows, per)
    assert n == rows * per
    for i in {0, per - 1, per, n // 2, (1 << 32) - 1, 1 << 32, n - per, n - 1}:
        if 0 <= i < n:
            assert (lib.item_row(rows, per, i), lib.item_tile(rows, per, i)) == (i // per, i % per)
