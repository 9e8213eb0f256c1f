"""Row kernels, scans and the small-join route at the sizes where they change
over, against the oracle.  Results are whole numbers: every comparison is
exact."""
import numpy as np
import pytest

from oracle import oracle_py as O

SHAPES = {
    # row widths (candidates a row), entries a row at most, z domain
    "packs": (list(range(1, 40)) + [127, 128, 129, 254, 255, 256, 257, 258, 339, 340, 341], 8, 100_000),
    "packs_many_entries": ([1, 3, 200, 256, 4095, 4096, 4097], 300, 100_000),
    "packs_bitmap_z": ([1, 31, 32, 33, 200, 256, 257, 700], 40, 300),
    "block_edges": ([1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096, 4097, 8191, 8192, 8193, 9000], 30, 262_144),
    "ranked_windows": ([300, 2500, 5000, 9000, 40_000], 200, 90_000),
    "one_row": ([20_000], 1500, 30_001),
}


def shape(name, reps=6, seed=3):
    """R (x, y) and S (z, y) whose rows have the widths of SHAPES[name]."""
    widths, ents, m = SHAPES[name]
    rng = np.random.default_rng(seed)
    R, S, y = [], [], 0
    for rep in range(1 if name == "one_row" else reps):
        for w in widths:
            n = min(w, 1 + (rep * ents) // reps if rep else 1) if name != "one_row" else ents
            cuts = np.sort(rng.integers(0, w + 1, n - 1))
            deg = np.diff(np.concatenate([[0], cuts, [w]]))
            x = rng.integers(0, 1 << 32)
            for d in deg:
                R.append((x, y))
                if d:
                    z = rng.choice(m, size=min(d, m), replace=False)
                    S.append(np.stack([z, np.full(z.shape[0], y)], 1))
                y += 1
    # every z of the domain occurs, joined by one more row and by none
    z = np.arange(m)
    S.append(np.stack([z, np.where(z % 3 == 0, y, y + 1)], 1))
    R.append((7, y))
    R = np.array(R, dtype=np.uint32)
    S = np.concatenate(S).astype(np.uint32)
    return R, S[rng.permutation(S.shape[0])]


def test_shapes_hold_their_widths():
    for name, (widths, ents, m) in SHAPES.items():
        R, S = shape(name)
        deg = np.bincount(S[:, 1], minlength=int(R[:, 1].max()) + 1)
        got = {}
        for x, y in R:
            got[x] = got.get(x, 0) + int(deg[y])
        assert set(min(w, m) for w in widths if w <= m) <= set(got.values()), name


def check(c, R, S, tag, ordered=False):
    want, n, _, _ = O.join_project(R, S)
    got = c.join_project(R, S)
    # the oracle always swaps a smaller R: its pairs are then (z, x)
    turned = c.get_param("keep_roles") and R.shape[0] < S.shape[0]
    want = want[:, ::-1] if turned else want
    assert got.shape[0] == n, tag
    assert np.array_equal(np.sort(O.pair_keys(got)), np.sort(O.pair_keys(want))), tag
    if ordered and n:
        x = got[:, 0]
        assert 1 + np.count_nonzero(x[1:] != x[:-1]) == np.unique(x).shape[0], tag
    wg, wc, ng, _, _ = O.join_count(R, S)
    wg = wg[:, ::-1] if turned else wg
    gp, gc = c.join_count(R, S)
    assert gp.shape[0] == ng, tag
    a, b = np.argsort(O.pair_keys(gp)), np.argsort(O.pair_keys(wg))
    assert np.array_equal(O.pair_keys(gp)[a], O.pair_keys(wg)[b]), tag
    assert np.array_equal(np.asarray(gc, np.uint64)[a], np.asarray(wc, np.uint64)[b]), tag


@pytest.mark.gpu
@pytest.mark.parametrize("prm", [{}, {"ordered_output": 1}, {"tile_bits_log2": 12}, {"tile_bits_log2": 12, "ordered_output": 1},
                                 {"block_slots_log2": 11, "warp_slots_log2": 7}, {"block_split": 0}, {"prefetch_rows": 1}],
                         ids=lambda p: ",".join(f"{k}={v}" for k, v in p.items()) or "default")
@pytest.mark.parametrize("name", SHAPES)
def test_row_widths(built, name, prm):
    """Packs, warp, block, bitmap and ranked rows at their limits, forked and
    alone, single pass and ordered, in one z tile and several."""
    import dim3gpu
    R, S = shape(name)
    c = dim3gpu.Context(0)
    for k, v in prm.items():
        c.set_param(k, v)
    c.set_param("keep_roles", 1)
    check(c, R, S, (name, prm), ordered="ordered_output" in prm)
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("prm", [{}, {"tile_bits_log2": 12}, {"dense_block": 0, "warp_slots_log2": 6, "block_slots_log2": 10}],
                         ids=lambda p: ",".join(f"{k}={v}" for k, v in p.items()) or "default")
@pytest.mark.parametrize("m", [9000, 32_768, 32_769, 98_305])
def test_count_rows_of_many_candidates(built, m, prm):
    """COUNT rows of 4096 and more candidates a tile, in the output and in the
    summaries, beside rows of a few and of one tile's."""
    import dim3gpu
    rng = np.random.default_rng(m)
    S = [np.stack([rng.choice(m, 8000, replace=False), np.full(8000, y)], 1) for y in range(40)]
    S = np.concatenate(S + [np.stack([np.arange(m), np.full(m, 40)], 1)]).astype(np.uint32)
    R = np.array([(x, y) for x in range(30) for y in range(40)] + [(77, 40), (78, 0), (79, 99)] +
                 [(100 + i, i % 40) for i in range(20)] + [(5, 7)] * 40, dtype=np.uint32)
    c = dim3gpu.Context(0)
    for k, v in {"keep_roles": 1, **prm}.items():
        c.set_param(k, v)
    check(c, R, S, (m, prm))
    import torch
    dR, dS = (torch.from_numpy(a.view(np.int32)).cuda() for a in (R, S))
    wg, wc, _, _, _ = O.join_count(R, S)
    want = O.tile_summary(np.ascontiguousarray(wg[:, ::-1]), wc, 4)  # the oracle's pairs are (z, x)
    assert np.array_equal(c.join_count_summary(dR, R.shape[0], dS, S.shape[0], 4), want)
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nx", [1, 2, 4095, 4096, 4097, 3 * 4096 + 1, 70_001])
def test_scan_tiles(built, nx):
    """Ids, row offsets and lists over prefix sums of one tile, its edges and
    several."""
    import dim3gpu
    rng = np.random.default_rng(nx)
    R = np.stack([np.arange(nx), rng.integers(0, nx, nx)], 1).astype(np.uint32)
    S = np.stack([np.arange(nx) * 3, rng.integers(0, nx, nx)], 1).astype(np.uint32)
    c = dim3gpu.Context(0)
    for ordered in (0, 1):
        c.set_param("ordered_output", ordered)
        check(c, R, S, (nx, ordered), ordered=bool(ordered))
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("keep", [0, 1])
@pytest.mark.parametrize("slack", [99, 150])
@pytest.mark.parametrize("nP,nQ", [(1, 1), (3, 900), (65_536, 65_536), (65_537, 65_536), (65_536, 65_537), (40_000, 65_536)])
def test_small_join_route_agrees(built, nP, nQ, slack, keep):
    """Joins of tuple-sized tables without a host round trip, and the general
    path on either side of the limit and below 100 % slack."""
    import dim3gpu
    rng = np.random.default_rng(nP + 2 * nQ)
    dom = max(1, max(nP, nQ) // 3)
    R = rng.integers(0, dom, (nP, 2)).astype(np.uint32)
    S = rng.integers(0, dom, (nQ, 2)).astype(np.uint32)
    c = dim3gpu.Context(0)
    c.set_param("table_slack_pct", slack)
    c.set_param("keep_roles", keep)
    for dense in (1, 0):
        c.set_param("dense_block", dense)
        check(c, R, S, (nP, nQ, slack, keep, dense))
        st = c.stats()
        assert st["swapped"] == (1 if nP < nQ and not keep else 0)
    # capacity is judged as on the general path
    _, n, _, _ = O.join_project(R, S)
    if n > 1:
        with pytest.raises(dim3gpu.Dim3GError) as e:
            c.join_project_into(R, S, np.empty((n - 1, 2), np.uint32))
        assert e.value.code == dim3gpu.ERR_CAPACITY
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nz", [1023, 1024, 1025, 4159])
@pytest.mark.parametrize("nx", [129, 255, 513])
def test_dense_emission_ragged(built, nx, nz):
    """Dense rows' pairs in whole lines: rows and columns off the tile sizes,
    lone pairs, full words and empty ones."""
    import dim3gpu
    rng = np.random.default_rng(nx * nz)
    A = rng.random((nx, 40)) < 0.3
    B = rng.random((40, nz)) < 0.2
    B[:, nz // 2:nz // 2 + 70] = False
    B[3, nz // 3:nz // 3 + 64] = True
    R = np.argwhere(A).astype(np.uint32)
    S = np.argwhere(B.T).astype(np.uint32)
    c = dim3gpu.Context(0)
    c.set_param("dense_block", 2)
    check(c, R, S, (nx, nz))
    c.close()


@pytest.mark.gpu
def test_noalloc_long_buckets(built):
    """Join values with thousands of tuples, duplicates and lone ones."""
    import ctypes

    import torch

    import dim3gpu
    rng = np.random.default_rng(8)
    hot = np.stack([rng.integers(0, 200, 5000), np.full(5000, 9)], 1)
    R = np.concatenate([hot, rng.integers(0, 30_000, (50_000, 2))]).astype(np.uint32)
    hot = np.stack([rng.integers(0, 2500, 3000), np.full(3000, 9)], 1)
    S = np.concatenate([hot, hot, rng.integers(0, 30_000, (40_000, 2))]).astype(np.uint32)
    want, n, _, _ = O.join_project(R, S)
    assert n < 1 << 20
    lib = dim3gpu.load()
    vp, u64 = ctypes.c_void_p, ctypes.c_uint64
    lib.dim3g_join_project_noalloc.argtypes = [vp, u64, vp, u64, vp, u64, ctypes.POINTER(u64), vp]
    dR, dS = (torch.from_numpy(a.view(np.int32)).cuda() for a in (R, S))
    out = torch.full((n, 2), -1, dtype=torch.int32, device="cuda")
    got = u64()
    for a, b, na, nb in ((dR, dS, R.shape[0], S.shape[0]),) * 2:
        rc = lib.dim3g_join_project_noalloc(vp(a.data_ptr()), na, vp(b.data_ptr()), nb, vp(out.data_ptr()), n,
                                            ctypes.byref(got), vp(torch.cuda.current_stream().cuda_stream))
        assert rc == dim3gpu.OK and got.value == n
        keys = O.pair_keys(out.cpu().numpy().view(np.uint32))
        assert np.array_equal(np.sort(keys), np.sort(O.pair_keys(want)))


@pytest.mark.gpu
def test_query_pass_row_widths(built):
    """One pass over relations of every row class, one of them empty."""
    import torch

    import dim3gpu
    host = [shape(n, reps=2) for n in SHAPES if n != "one_row"]
    host.append((np.zeros((0, 2), np.uint32), np.array([[1, 2]], np.uint32)))
    c = dim3gpu.Context(0)
    dev = [torch.from_numpy(a.view(np.int32)).cuda() if a.shape[0] else 0 for h in host for a in h]
    rs = dim3gpu.RelSet(c, [(d, a.shape[0]) for d, a in zip(dev, [a for h in host for a in h])])
    specs, want = [], []
    for k, (R, S) in enumerate(host):
        for op in (dim3gpu.OP_PROJECT, dim3gpu.OP_COUNT):
            w = O.join_project(R, S)[0] if op == dim3gpu.OP_PROJECT else O.join_count(R, S)[:2]
            n = (w if op == dim3gpu.OP_PROJECT else w[0]).shape[0]
            s = {"r": 2 * k, "s": 2 * k + 1, "op": op, "capacity": n,
                 "out": torch.empty((max(n, 1), 2), dtype=torch.int32, device="cuda")}
            if op == dim3gpu.OP_COUNT:
                s["cnt"] = torch.empty((max(n, 1),), dtype=torch.int64, device="cuda")
            specs.append(s)
            want.append(w)
    for _ in range(2):
        res = rs.join(specs)
        torch.cuda.synchronize()
        for s, r, w in zip(specs, res, want):
            pairs = w if s["op"] == dim3gpu.OP_PROJECT else w[0]
            assert r["n_out"] == pairs.shape[0]
            k = O.pair_keys(s["out"][:r["n_out"]].cpu().numpy().view(np.uint32))
            a, b = np.argsort(k), np.argsort(O.pair_keys(pairs))
            assert np.array_equal(k[a], O.pair_keys(pairs)[b])
            if s["op"] == dim3gpu.OP_COUNT:
                got = s["cnt"][:r["n_out"]].cpu().numpy().view(np.uint64)
                assert np.array_equal(got[a], np.asarray(w[1], np.uint64)[b])
    rs.close()
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("ordered", [0, 1])
def test_few_block_rows_get_the_full_cta_width(built, ordered):
    """120 rows of a million candidates over 1000 z: split by set size, they take
    no longer than in one launch of full-width CTAs (time against time)."""
    import torch

    import dim3gpu
    rng = np.random.default_rng(9)
    R = np.stack([np.repeat(np.arange(120), 1000), np.tile(np.arange(1000), 120)], 1).astype(np.uint32)
    S = np.stack([rng.integers(0, 1000, 1_000_000), rng.integers(0, 1000, 1_000_000)], 1).astype(np.uint32)
    dR, dS = (torch.from_numpy(a.view(np.int32)).cuda() for a in (R, S))
    out = torch.empty((120 * 1000, 2), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ms = []
    for split in (0, 1):
        c = dim3gpu.Context(0)
        for k, v in dict(keep_roles=1, ordered_output=ordered, block_split=split).items():
            c.set_param(k, v)
        best = 1e9
        for _ in range(6):
            assert c.join_project_device(dR, R.shape[0], dS, S.shape[0], out, out.shape[0]) == out.shape[0]
            best = min(best, c.stats()["ms_write"])
        assert c.stats()["rows_block"] == 120
        ms.append(best)
        c.close()
    assert ms[1] < 1.2 * ms[0] + 0.02, ms
