"""Device memory that relation sets, batches and servers report and hold
themselves to: COUNT's counters (a word a z of one tile and SM) among it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE = 1 << 19  # default z tile


def counters():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count * TILE * 4


def relations(n=3000):
    import torch
    rng = np.random.default_rng(4)
    return [(torch.from_numpy(rng.integers(0, 500, (n, 2)).astype(np.int32)).cuda(), n) for _ in range(2)]


def outputs(op, cap=400_000):
    import torch
    return {"r": 0, "s": 1, "op": op, "capacity": cap, "out": torch.empty((cap, 2), dtype=torch.int32, device="cuda"),
            "cnt": torch.empty(cap, dtype=torch.int64, device="cuda")}


def test_relation_set_reports_count_scratch(ctx):
    import dim3gpu
    rs = dim3gpu.RelSet(ctx, relations())
    rs.join([outputs(dim3gpu.OP_PROJECT)])
    before = rs.bytes()
    rs.join([outputs(dim3gpu.OP_COUNT)])
    assert rs.bytes() == before + counters()
    rs.close()


def test_batch_reports_count_scratch(ctx):
    import dim3gpu
    got = []
    for op in (dim3gpu.OP_PROJECT, dim3gpu.OP_COUNT):
        b = dim3gpu.Batch(ctx, [tuple(relations())], [outputs(op)])
        b.run()
        got.append(b.info()["device_bytes"])
        b.close()
    assert got[1] == got[0] + counters()


@pytest.mark.parametrize("lanes", [1, 3])
def test_server_budget_holds_its_lanes(ctx, lanes):
    """budget_bytes covers the set and the lanes' scratch, as the device sees
    it: a budget that does not is refused."""
    import torch

    import dim3gpu
    rs = dim3gpu.RelSet(ctx, relations())
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    srv = dim3gpu.Server(rs, lanes=lanes, max_batch=4, budget_bytes=1 << 45)
    used = free - torch.cuda.mem_get_info()[0]
    fixed = (1 << 45) - srv.stats()["output_budget"]
    srv.close()
    assert used >= lanes * counters()
    assert fixed + (64 << 20) >= rs.bytes() + used  # 64 MB: streams and allocation granules
    with pytest.raises(dim3gpu.Dim3GError) as e:
        dim3gpu.Server(rs, lanes=lanes, max_batch=4, budget_bytes=fixed - 1)
    assert e.value.code == dim3gpu.ERR_NOMEM
    dim3gpu.Server(rs, lanes=lanes, max_batch=4, budget_bytes=fixed + 4096).close()
    rs.close()
