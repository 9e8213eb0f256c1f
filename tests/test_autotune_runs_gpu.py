"""dim3g_autotune's max_trials bounds the joins that it runs: one pass for the
output's size, and two runs a trial."""
import numpy as np
import pytest


@pytest.mark.gpu
def test_autotune_runs_no_more_than_its_trials(built):
    import torch

    import dim3gpu
    rng = np.random.default_rng(5)
    # 40 rows of about 30K candidates over 120K z: bitmap rows, too few for the product
    R = np.stack([rng.integers(0, 40, 20_000), rng.integers(0, 2000, 20_000)], 1)
    S = np.stack([np.arange(120_000), rng.integers(0, 2000, 120_000)], 1)
    dR, dS = (torch.from_numpy(a.astype(np.int32)).cuda() for a in (R, S))
    c = dim3gpu.Context(0)
    c.set_param("keep_roles", 1)

    def launches(call):
        before = c.stats()["launches"]
        call()
        return c.stats()["launches"] - before

    a = (dR, R.shape[0], dS, S.shape[0])
    size = launches(lambda: c.join_project_count_device(*a))
    n = c.join_project_count_device(*a)
    out = torch.empty((n, 2), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    run = {}
    for dense in (0, 1):
        c.set_param("dense_block", dense)
        run[dense] = launches(lambda: c.join_project_device(*a, out, n))
    assert c.stats()["rows_bitmap"] > 0 and c.stats()["rows_dense"] == 0
    got = launches(lambda: c.autotune(*a, max_trials=2))
    assert got == size + 2 * run[1] + 2 * run[0]
    c.close()
