"""First values of very many tuples (hubs): their rows are worked out by more
than one warp.  Results against the oracle, exact; times only as ratios of
parts of one call."""
import numpy as np
import pytest

from oracle import oracle_py as O

pytestmark = pytest.mark.gpu

# entries of the long rows: about the lengths at which a row goes to the CTA,
# or to the whole grid in pieces
LENGTHS = [2047, 2048, 2049, 4096, 4097, 8191, 8192, 8193, 10_241, 20_000]


def hubs(lengths, short, seed):
    """R: row x of lengths[x] entries, and `short` rows of two; S: a few tuples
    for every fifth join value."""
    rng = np.random.default_rng(seed)
    n_y = 30_000
    R = [np.stack([np.full(k, x), rng.choice(n_y, k, replace=False)], 1) for x, k in enumerate(lengths)]
    R.append(np.stack([1000 + np.arange(2 * short) // 2, rng.integers(0, n_y, 2 * short)], 1))
    R = np.concatenate(R).astype(np.uint32)
    S = np.stack([rng.integers(0, 3000, n_y), 5 * rng.integers(0, n_y // 5, n_y)], 1).astype(np.uint32)
    return R[rng.permutation(R.shape[0])], S


@pytest.mark.parametrize("ordered", [0, 1])
@pytest.mark.parametrize("lengths,short", [(LENGTHS, 30_000), ([2100] * 40, 0), ([20_000], 0), ([3000] * 9, 5)])
def test_join_with_hubs(ctx, lengths, short, ordered):
    R, S = hubs(lengths, short, len(lengths))
    import dim3gpu
    c = dim3gpu.Context(0)
    c.set_param("ordered_output", ordered)
    c.set_param("keep_roles", 1)
    want = O.join_project(R, S)[0]
    wg, wc = O.join_count(R, S)[:2]
    if R.shape[0] < S.shape[0]:  # the oracle swaps
        want, wg = want[:, ::-1], wg[:, ::-1]
    assert np.array_equal(np.sort(O.pair_keys(c.join_project(R, S))), np.sort(O.pair_keys(want)))
    assert c.stats()["out_j"] == int(wc.sum())
    gp, gc = c.join_count(R, S)
    a, b = np.argsort(O.pair_keys(gp)), np.argsort(O.pair_keys(wg))
    assert np.array_equal(O.pair_keys(gp)[a], O.pair_keys(wg)[b]) and np.array_equal(gc[a], np.asarray(wc)[b])
    c.close()


def star(n, hub):
    """Device R with one first value of `hub` tuples among n, S uniform."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(6)
    n_y = n * 3 // 4

    def ints(hi, k):
        return torch.randint(0, hi, (k,), generator=g, device="cuda")

    x = torch.cat([torch.full((hub,), 7, device="cuda"), ints(n // 4, n - hub)])
    y = torch.cat([torch.randperm(n_y, generator=g, device="cuda")[:hub], ints(n_y, n - hub)])
    p = torch.randperm(n, generator=g, device="cuda")
    R = torch.stack([x[p], y[p]], 1).to(torch.int32).contiguous()
    S = torch.stack([ints(n // 8, n - 1000), ints(n_y, n - 1000)], 1).to(torch.int32).contiguous()
    return R, S


def test_hub_row_is_binned_in_less_than_its_expansion(ctx):
    """One CTA expands the hub's row; counting its candidates beforehand, in a
    warp, took longer than that."""
    import torch
    R, S = star(4_000_000, 2_000_000)
    out = torch.empty((16_000_000, 2), dtype=torch.int32, device="cuda")
    best = {}
    for _ in range(3):
        ctx.join_project_device(R, R.shape[0], S, S.shape[0], out, out.shape[0])
        st = ctx.stats()
        for k in ("ms_csr", "ms_write"):
            best[k] = min(best.get(k, 1e9), st[k])
    assert best["ms_csr"] < best["ms_write"], best
