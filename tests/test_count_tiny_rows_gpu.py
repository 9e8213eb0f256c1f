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
