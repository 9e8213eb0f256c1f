"""Results and work past 2^32: sizes of results that no buffer holds, and the
places of a result's rows in it.  Every x joins every z, so the sizes are
products; every comparison is exact."""
import ctypes

import numpy as np
import pytest

NX, NZ = 4200, 1_100_000  # more than 2^32 pairs in one 4096-row tile of the prefix sum


def ready(*t):
    """The library runs on streams of its own."""
    import torch
    torch.cuda.synchronize()
    return t


def all_pairs():
    import torch
    x = torch.arange(NX, dtype=torch.int32, device="cuda")
    z = torch.randperm(NZ, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").to(torch.int32)
    return ready(torch.stack([x, torch.zeros_like(x)], 1).contiguous(), torch.stack([z, torch.zeros_like(z)], 1).contiguous())


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
    out, cnt = ready(torch.full((cap, 2), -5, dtype=torch.int32, device="cuda"),
                     torch.full((cap,), -5, dtype=torch.int64, device="cuda"))
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


WIDE_Z = 9000  # a bitmap row of one tile


def wide_row(pad):
    """R: 1024 times (3, 0), and pad tuples without a partner; S: 2^22 - 1
    tuples of WIDE_Z values.  Row 3 has 2^32 - 1024 candidates, in one tile."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(2)
    z = torch.randint(0, WIDE_Z, ((1 << 22) - 1,), generator=g, device="cuda", dtype=torch.int32)
    x = torch.full((1024 + pad,), 3, dtype=torch.int32, device="cuda")
    y = torch.zeros_like(x)
    x[1024:], y[1024:] = 4, 1
    mult = torch.bincount(z.to(torch.int64), minlength=WIDE_Z)
    assert 1024 * int(mult.sum()) == (1 << 32) - 1024 and int(mult.min()) > 0
    return ready(torch.stack([x, y], 1).contiguous(), torch.stack([z, torch.zeros_like(z)], 1).contiguous(), 1024 * mult)


def check_wide(out, cnt, n, mult):
    assert n == WIDE_Z and bool((out[:n, 0] == 3).all())
    z = out[:n, 1].to("cpu").numpy()
    assert np.array_equal(np.sort(z), np.arange(WIDE_Z))
    assert cnt is None or np.array_equal(cnt[:n].cpu().numpy(), mult.cpu().numpy()[z])


@pytest.mark.gpu
@pytest.mark.parametrize("count", [0, 1])
def test_row_of_almost_2_32_candidates(built, count):
    """One join: the whole-tile bitmap row, and COUNT's counter a z."""
    import torch
    R, S, mult = wide_row(0)
    out = torch.empty((WIDE_Z, 2), dtype=torch.int32, device="cuda")
    cnt = torch.empty(WIDE_Z, dtype=torch.int64, device="cuda") if count else None
    c = context(dense_block=0)
    a = (R, R.shape[0], S, S.shape[0], out)
    n = c.join_count_device(*a, cnt, WIDE_Z) if count else c.join_project_device(*a, WIDE_Z)
    check_wide(out, cnt, n, mult)
    c.close()


@pytest.mark.gpu
def test_query_row_of_almost_2_32_candidates(built):
    """A query pass: the bitmap row and the ranked row."""
    import torch

    import dim3gpu
    R, S, mult = wide_row(1 << 22)
    c = dim3gpu.Context(0)
    rs = dim3gpu.RelSet(c, [(R, R.shape[0]), (S, S.shape[0])])
    outs = [torch.empty((WIDE_Z, 2), dtype=torch.int32, device="cuda") for _ in range(2)]
    cnt = torch.empty(WIDE_Z, dtype=torch.int64, device="cuda")
    got = rs.join([{"r": 0, "s": 1, "op": op, "out": outs[op], "cnt": cnt, "capacity": WIDE_Z}
                   for op in (dim3gpu.OP_PROJECT, dim3gpu.OP_COUNT)])
    for op, r in enumerate(got):
        assert r["out_j"] == (1 << 32) - 1024
        check_wide(outs[op], cnt if op else None, r["n_out"], mult)
    rs.close()
    c.close()


@pytest.mark.gpu
def test_sizes_around_the_wide_sums(built):
    """Rows of 2^20 - 1 and 2^20 pairs: on either side of where a tile's sum
    can pass 2^32, alone and in one result."""
    import torch
    nz = 1 << 20
    z = torch.arange(nz, dtype=torch.int32, device="cuda")
    S = torch.cat([torch.stack([z, torch.zeros_like(z)], 1), torch.stack([z[1:], torch.ones_like(z[1:])], 1)]).contiguous()
    c = context(dense_block=0)
    for ys in ([0] * 4096, [1] * 4096, [1] * 4096 + [0] + [1] * 4095, [1] * 5000 + [2] * 5000 + [0] * 3000):
        R, = ready(torch.tensor([[x, y] for x, y in enumerate(ys)], dtype=torch.int32, device="cuda"))
        n = sum({0: nz, 1: nz - 1, 2: 0}[y] for y in ys)
        assert c.join_project_count_device(R, len(ys), S, S.shape[0]) == n
    c.close()


@pytest.mark.gpu
def test_count_over_wide_domains_takes_any_tile_width(built):
    """1.2M join values and 4M z: 2^32 row pointers at 2^10 z a tile, which
    COUNT does not need."""
    import torch
    ny, nz = 1_200_000, 4_000_000
    y, z = torch.arange(ny, device="cuda"), torch.arange(nz, device="cuda")
    R, S = ready(torch.stack([y % 1000, y], 1).to(torch.int32).contiguous(),
                 torch.stack([z, z % ny], 1).to(torch.int32).contiguous())
    out = torch.empty((nz, 2), dtype=torch.int32, device="cuda")
    cnt = torch.empty(nz, dtype=torch.int64, device="cuda")
    c = context(tile_bits_log2=10)
    assert ny * (nz >> 10) >= 1 << 32
    assert c.join_count_device(R, ny, S, nz, out, cnt, nz) == nz
    assert bool((cnt == 1).all())
    order = torch.argsort(out[:, 1])
    assert torch.equal(out[order, 1].long(), z) and torch.equal(out[order, 0].long(), (z % ny) % 1000)
    assert c.stats()["z_tiles"] <= 1 << 9
    c.close()
