"""The ordered write pass' own check of a row's count, on the kernel alone
(through the library the counts are the count pass' and always fit)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "joinproject-dim3_gb300", "csrc")

SRC = r"""
#include "ordered.cuh"
using namespace dim3g;
// Two tiny rows of one entry each, n0 and n1 pairs, written at off0 and off1
// as if they had cnt0 and cnt1.  out: 64 pairs, as the caller filled them.
extern "C" int write_rows(uint32_t n0, uint32_t n1, uint32_t cnt0, uint32_t cnt1, uint64_t off0, uint64_t off1, uint32_t* out) {
    struct All {
        uint32_t JR_R[3], IC_R[2], JR_S[3], id2x[2], ucap[2], cnt[2], rows[2], err;
        unsigned long long off[2], nrows;
        uint2 ISV[64], out[64];
    };
    All h{{0, 1, 2}, {0, 1}, {0, n0, n0 + n1}, {100, 101}, {n0, n1}, {cnt0, cnt1}, {0, 1}, 0, {off0, off1}, 2, {}, {}};
    for (uint32_t i = 0; i < n0 + n1; i++) h.ISV[i] = make_uint2(i < n0 ? i : i - n0, 1000 + (i < n0 ? i : i - n0));
    memcpy(h.out, out, sizeof h.out);
    All* d = nullptr;
    if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMemcpy(d, &h, sizeof h, cudaMemcpyHostToDevice) != cudaSuccess) return -1;
    RowCtx c{};
    c.JR_R = d->JR_R, c.IC_R = d->IC_R, c.JR_S = d->JR_S, c.ISV = d->ISV, c.T = 1, c.tile_width = c.m = 32;
    c.ucap = d->ucap, c.cnt = d->cnt, c.off = d->off, c.id2x = d->id2x, c.out = d->out, c.err = &d->err;
    const int smem = (int)(8 * kRowsPackWords * 4);
    if (cudaFuncSetAttribute(k_rows_pack<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -1;
    k_rows_pack<true><<<1, 256, smem>>>(c, d->rows, &d->nrows);
    if (cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    cudaFree(d);
    memcpy(out, h.out, sizeof h.out);
    return (int)h.err;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    import build
    d = tmp_path_factory.mktemp("rows")
    src, so = str(d / "rows.cu"), str(d / "rows.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run([build._nvcc()] + build.NVCC_FLAGS + ["-shared", "-I", CSRC, src, "-o", so], check=True)
    L = ctypes.CDLL(so)
    L.write_rows.argtypes = [ctypes.c_uint32] * 4 + [ctypes.c_uint64] * 2 + [ctypes.c_void_p]
    return L


@pytest.mark.gpu
@pytest.mark.parametrize("n0,n1,cnt0,cnt1", [(5, 7, 5, 7), (5, 7, 3, 7), (5, 7, 5, 0), (32, 1, 31, 1), (4, 4, 6, 4)])
def test_packed_rows_stay_in_their_counts(lib, n0, n1, cnt0, cnt1):
    out = np.full((64, 2), 7, np.uint32)
    off0, off1 = 3, 3 + cnt0 + 2
    err = lib.write_rows(n0, n1, cnt0, cnt1, off0, off1, out.ctypes.data)
    assert err == (0 if (n0, n1) == (cnt0, cnt1) else 4)  # kErrOutputBound
    touched = np.zeros(64, bool)
    for x, n, cnt, off in ((100, n0, cnt0, off0), (101, n1, cnt1, off1)):
        k = min(n, cnt)
        touched[off:off + k] = True
        assert (out[off:off + k, 0] == x).all()
        z = out[off:off + k, 1]
        assert np.unique(z).shape[0] == k and (z >= 1000).all() and (z < 1000 + n).all()
    assert (out[~touched] == 7).all()
