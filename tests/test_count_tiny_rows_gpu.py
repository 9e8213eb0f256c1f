"""COUNT rows of a few candidates at exact offsets and in summaries: results
against the single pass', and time against it."""
import numpy as np
import pytest

from oracle import oracle_py as O

pytestmark = pytest.mark.gpu


def relations(n_x, m, seed, n_y=14_000, deg=5):
    rng = np.random.default_rng(seed)
    R = np.stack([rng.integers(0, n_x, 4 * n_x), rng.integers(0, n_y, 4 * n_x)], 1).astype(np.uint32)
    S = np.stack([rng.integers(0, m, n_y * deg), rng.integers(0, n_y, n_y * deg)], 1).astype(np.uint32)
    return R, S


@pytest.mark.parametrize("m", [3, 100, 257, 1025, 60_000])
def test_tiny_count_rows_at_offsets_and_in_summaries(ctx, m):
    import torch

    import dim3gpu
    R, S = relations(20_000, m, m)
    wg, wc = O.join_count(R, S)[:2]
    c = dim3gpu.Context(0)
    c.set_param("ordered_output", 1)
    gp, gc = c.join_count(R, S)
    a, b = np.argsort(O.pair_keys(gp)), np.argsort(O.pair_keys(wg))
    assert np.array_equal(O.pair_keys(gp)[a], O.pair_keys(wg)[b]) and np.array_equal(gc[a], np.asarray(wc)[b])
    assert 1 + np.count_nonzero(gp[1:, 0] != gp[:-1, 0]) == np.unique(gp[:, 0]).shape[0]
    dR, dS = (torch.from_numpy(r.view(np.int32)).cuda() for r in (R, S))
    torch.cuda.synchronize()
    assert np.array_equal(c.join_count_summary(dR, R.shape[0], dS, S.shape[0], 4), O.tile_summary(wg, wc, 4))
    c.close()


def test_tiny_count_rows_take_no_cta_each(ctx):
    """500K rows of 20 candidates: with a CTA a row the summary took twelve times
    the single pass' rows."""
    import torch
    R, S = relations(500_000, 100, 1)
    dR, dS = (torch.from_numpy(r.view(np.int32)).cuda() for r in (R, S))
    cap = 12_000_000
    out = torch.empty((cap, 2), dtype=torch.int32, device="cuda")
    cnt = torch.empty(cap, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    a = (dR, R.shape[0], dS, S.shape[0])
    ms = []
    for call in (lambda: ctx.join_count_device(*a, out, cnt, cap), lambda: ctx.join_count_summary(*a, 1)):
        best = 1e9
        for _ in range(5):
            call()
            best = min(best, ctx.stats()["ms_write"])
        ms.append(best)
    assert ms[1] < 5 * ms[0], ms


@pytest.mark.parametrize("n_y,m,n_s", [(31, 80, 62_000), (400, 250, 45_000), (9, 3, 36_000), (40, 5000, 4100)])
def test_packs_of_long_segments(ctx, n_y, m, n_s):
    """Tiny rows of one to three entries with a hundred to four thousand
    candidates each, beside join values with few: every form of a join and a
    pass over resident relations."""
    import torch

    import dim3gpu
    rng = np.random.default_rng(n_y)
    R = np.stack([rng.integers(0, 20_000, 30_000), rng.integers(0, n_y + 5, 30_000)], 1).astype(np.uint32)
    S = np.stack([rng.integers(0, m, n_s), rng.integers(0, n_y, n_s)], 1)
    S = np.concatenate([S, [[1, n_y], [2, n_y + 1], [m + 7, n_y + 2]]]).astype(np.uint32)
    for ordered in (0, 1):
        c = dim3gpu.Context(0)
        c.set_param("ordered_output", ordered)
        c.set_param("keep_roles", 1)
        want, wg, wc = O.join_project(R, S)[0], *O.join_count(R, S)[:2]
        if R.shape[0] < S.shape[0]:  # the oracle swaps
            want, wg = want[:, ::-1], wg[:, ::-1]
        assert np.array_equal(np.sort(O.pair_keys(c.join_project(R, S))), np.sort(O.pair_keys(want)))
        gp, gc = c.join_count(R, S)
        a, b = np.argsort(O.pair_keys(gp)), np.argsort(O.pair_keys(wg))
        assert np.array_equal(O.pair_keys(gp)[a], O.pair_keys(wg)[b]) and np.array_equal(gc[a], np.asarray(wc)[b])
        c.close()
    pad = np.stack([np.arange(40_000) + 50_000, np.full(40_000, n_y + 99)], 1).astype(np.uint32)
    R2 = np.concatenate([R, pad])  # R drives the pass
    dev = [torch.from_numpy(r.view(np.int32)).cuda() for r in (R2, S)]
    rs = dim3gpu.RelSet(ctx, [(d, d.shape[0]) for d in dev])
    wg, wc = O.join_count(R2, S)[:2]
    n = wg.shape[0]
    out = [torch.empty((n, 2), dtype=torch.int32, device="cuda") for _ in range(2)]
    cnt = torch.empty(n, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    got = rs.join([{"r": 0, "s": 1, "op": op, "out": out[op], "cnt": cnt, "capacity": n} for op in (0, 1)])
    b = np.argsort(O.pair_keys(wg))
    for op in (0, 1):
        assert got[op]["n_out"] == n
        k = O.pair_keys(out[op].cpu().numpy().view(np.uint32))
        a = np.argsort(k)
        assert np.array_equal(k[a], O.pair_keys(wg)[b])
    assert np.array_equal(cnt.cpu().numpy().view(np.uint64)[a], np.asarray(wc)[b])
    rs.close()
