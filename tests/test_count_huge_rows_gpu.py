"""COUNT rows of very many groups beside many middling ones (so that the rows
are ranked, not counted directly): in one z tile and several, in the output, at
exact offsets and in summaries."""
import numpy as np
import pytest

from oracle import oracle_py as O

pytestmark = pytest.mark.gpu


def relations(m, n_mid, huge, seed):
    """R (x, y), S (z, y): n_mid rows of 2500 candidates over m z, and one row
    of every width in `huge`, all of its z distinct but for a few."""
    rng = np.random.default_rng(seed)
    n_y, deg, ent = 4000, 20, 125
    R = [np.stack([np.repeat(np.arange(n_mid), ent), rng.integers(0, n_y, n_mid * ent)], 1)]
    S = [np.stack([rng.integers(0, m, n_y * deg), np.repeat(np.arange(n_y), deg)], 1)]
    for k, w in enumerate(huge):
        R.append(np.array([[n_mid + k, n_y + k]] * (1 + k % 2) + [[n_mid + k, 7]]))
        S.append(np.stack([rng.choice(m, w, replace=False), np.full(w, n_y + k)], 1))
    R, S = np.concatenate(R).astype(np.uint32), np.concatenate(S).astype(np.uint32)
    return R, S[rng.permutation(S.shape[0])]


@pytest.mark.parametrize("prm", [{}, {"ordered_output": 1}, {"tile_bits_log2": 17}, {"tile_bits_log2": 17, "ordered_output": 1}],
                         ids=lambda p: ",".join(f"{k}={v}" for k, v in p.items()) or "default")
@pytest.mark.parametrize("m,huge", [(150_000, [65_537, 150_000]), (200_000, [70_000, 199_999, 90_000]), (600_000, [600_000, 100_000])])
def test_huge_rows_among_ranked_ones(ctx, m, huge, prm):
    import torch

    import dim3gpu
    R, S = relations(m, 300, huge, m)
    wg, wc = O.join_count(R, S)[:2]
    if R.shape[0] < S.shape[0]:  # the oracle swaps
        wg = wg[:, ::-1]
    c = dim3gpu.Context(0)
    for k, v in dict(keep_roles=1, **prm).items():
        c.set_param(k, v)
    dR, dS = (torch.from_numpy(a.view(np.int32)).cuda() for a in (R, S))
    n = wg.shape[0]
    out = torch.empty((n, 2), dtype=torch.int32, device="cuda")
    cnt = torch.empty(n, dtype=torch.int64, device="cuda")
    b = np.argsort(O.pair_keys(wg))
    for _ in range(2):
        assert c.join_count_device(dR, R.shape[0], dS, S.shape[0], out, cnt, n) == n
        k = O.pair_keys(out.cpu().numpy().view(np.uint32))
        a = np.argsort(k)
        assert np.array_equal(k[a], O.pair_keys(wg)[b])
        assert np.array_equal(cnt.cpu().numpy().view(np.uint64)[a], np.asarray(wc)[b])
    want = O.tile_summary(np.ascontiguousarray(wg), wc, 4)
    assert np.array_equal(c.join_count_summary(dR, R.shape[0], dS, S.shape[0], 4), want)
    c.close()


def test_one_huge_row_does_not_hold_up_the_others(ctx):
    """A row of every z: counted in windows of ranks, its CTA walked it 25 times
    while the rest of the GPU was done."""
    import torch

    import dim3gpu
    c = dim3gpu.Context(0)
    c.set_param("keep_roles", 1)
    ms = []
    for huge in ([], [200_000]):
        R, S = relations(200_000, 2000, huge, 1)
        dR, dS = (torch.from_numpy(a.view(np.int32)).cuda() for a in (R, S))
        cap = 2000 * 2600 + 300_000
        out = torch.empty((cap, 2), dtype=torch.int32, device="cuda")
        cnt = torch.empty(cap, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        best = 1e9
        for _ in range(5):
            c.join_count_device(dR, R.shape[0], dS, S.shape[0], out, cnt, cap)
            best = min(best, c.stats()["ms_write"])
        ms.append(best)
    assert c.stats()["rows_bitmap"] > 2000  # the rows are not map rows
    assert ms[1] < 2 * ms[0] + 0.4, ms
    c.close()
