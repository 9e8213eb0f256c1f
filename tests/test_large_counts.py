"""Results and work past 2^32: sizes of results that no buffer holds, and the
places of a result's rows in it.  Every x joins every z, so the sizes are
products; every comparison is exact."""
import ctypes

import numpy as np
import pytest

NX, NZ = 4200, 1_100_000  # more than 2^32 pairs in one 4096-row tile of the prefix sum


def all_pairs():
    import torch
    x = torch.arange(NX, dtype=torch.int32, device="cuda")
    z = torch.randperm(NZ, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").to(torch.int32)
    return (torch.stack([x, torch.zeros_like(x)], 1).contiguous(), torch.stack([z, torch.zeros_like(z)], 1).contiguous())


def context(**prm):
    import dim3gpu
    c = dim3gpu.Context(0)
    for k, v in dict(keep_roles=1, **prm).items():
        c.set_param(k, v)
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("dense", [0, 1, 2])
def test_size_of_a_result_past_2_32(built, dense):
    """The count pass' total, from the row kernels and from the product."""
    R, S = all_pairs()
    c = context(dense_block=dense)
    assert c.join_project_count_device(R, NX, S, NZ) == NX * NZ
    assert dense < 2 or c.stats()["rows_dense"] == NX
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dense", [0, 2])
@pytest.mark.parametrize("count", [0, 1])
def test_ordered_result_past_2_32_is_refused(built, count, dense):
    """A buffer that cannot hold the result: its size, nothing written."""
    import torch

    import dim3gpu
    R, S = all_pairs()
    c = context(ordered_output=1, dense_block=dense)
    cap = 1024
    out = torch.full((cap, 2), -5, dtype=torch.int32, device="cuda")
    cnt = torch.full((cap,), -5, dtype=torch.int64, device="cuda")
    n = ctypes.c_uint64()
    L, p = dim3gpu.load(), ctypes.c_void_p
    if count:
        rc = L.dim3g_join_count_device(c.h, p(R.data_ptr()), NX, p(S.data_ptr()), NZ, p(out.data_ptr()), p(cnt.data_ptr()), cap,
                                       ctypes.byref(n))
    else:
        rc = L.dim3g_join_project_device(c.h, p(R.data_ptr()), NX, p(S.data_ptr()), NZ, p(out.data_ptr()), cap, ctypes.byref(n))
    assert rc == dim3gpu.ERR_CAPACITY and n.value == NX * NZ
    assert bool((out == -5).all()) and bool((cnt == -5).all())
    c.close()


@pytest.mark.gpu
def test_ordered_rows_past_2_32(built):
    """The whole ordered result where it fits (37 GB): every row's pairs at its
    own offset, in x-id order."""
    import torch
    R, S = all_pairs()
    if torch.cuda.mem_get_info()[0] < 8 * NX * NZ + (16 << 30):
        pytest.skip("the result does not fit this device")
    c = context(ordered_output=1)
    out = torch.empty((NX * NZ, 2), dtype=torch.int32, device="cuda")
    assert c.join_project_device(R, NX, S, NZ, out, NX * NZ) == NX * NZ
    want = NZ * (NZ - 1) // 2
    seen = set()
    for r in range(NX):
        rows = out[r * NZ:(r + 1) * NZ]
        seen.add(int(rows[0, 0]))
        if r % 64 == 0 or r == NX - 1:
            assert bool((rows[:, 0] == rows[0, 0]).all()) and int(rows[:, 1].sum(dtype=torch.int64)) == want, r
    assert seen == set(range(NX))
    c.close()


def test_sizes_used_here():
    assert 4096 * NZ >= 1 << 32 and np.iinfo(np.uint32).max < NX * NZ
