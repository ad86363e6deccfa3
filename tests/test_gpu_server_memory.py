"""A server takes its device memory when it is made: batches of whatever size
allocate none while it serves, and answer the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_no_allocation_while_serving(gpu_ctx):
    import torch
    import libfastlib_b200 as L
    from libfastlib_b200 import workloads as W
    n = 4_000_003
    cols = [L.Index.build(gpu_ctx, L.RELIC, W.uniform_int_column(c, n, 1000)) for c in range(3)]
    metas = [{"kind": "relic", "card": 1000}] * 3
    qs = W.conjunctive_queries(8, metas, 1500, max_terms=3)
    queries = [[cols[c].term(lo, hi) for c, lo, hi in q] for q in qs]
    rng = np.random.default_rng(8)
    want = None
    for made in range(2):  # the kernels are loaded by the first
        S = L.Server(gpu_ctx, nslots=3, max_batch=512, scratch_budget=1 << 29)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        for rate in (2000, 20_000, 200_000, 2_000_000):
            counts, lat, wall, ids = S.replay(queries, np.cumsum(rng.exponential(1 / rate, len(queries))), rid_cap=600)
            if want is None:
                want = [int(c) for c in counts]
            assert [int(c) for c in counts] == want
        if made:
            assert torch.cuda.mem_get_info()[0] == free
        S.close()
    for q in range(0, 1500, 100):
        c, rids, _ = L.evaluate(gpu_ctx, queries[q])
        assert c == want[q] and np.array_equal(ids[q], rids[:600])
    for x in cols:
        x.close()
