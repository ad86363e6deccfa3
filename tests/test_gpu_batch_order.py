"""The default order of a batch with row ids: one pass where all ids are wanted
or most tiles hold ids under the limits, two passes for a large batch whose
limits leave most tiles unvisited; the ids are the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,caps,passes", [(400, None, 1), (400, 5, 3), (400, 1 << 20, 1), (40, 5, 1)])
def test_passes(nq, caps, passes):
    import libfastlib_b200 as L
    ctx = L.Context(0)
    n = 1_000_003  # 8 tiles a query
    rng = np.random.default_rng(nq)
    vals = rng.integers(0, 100, n).astype(np.uint32)
    idx = L.Index.build(ctx, L.RELIC, vals)
    spans = [tuple(sorted(rng.choice(101, 2, replace=False))) for _ in range(nq)]
    want = [np.flatnonzero((vals >= a) & (vals < b)) for a, b in spans]
    terms = [[idx.term(float(a), float(b))] for a, b in spans]
    if caps is None:
        B = L.Batch(ctx, terms, rid_cap=sum(len(w) for w in want))
    else:
        B = L.Batch(ctx, terms, caps=[caps] * nq)
    for _ in range(2):
        l0 = ctx.launches
        B.run()
        assert ctx.launches - l0 == passes
    assert B.counts().tolist() == [len(w) for w in want]
    for q in range(0, nq, 7):
        k = len(want[q]) if caps is None else min(caps, len(want[q]))
        assert np.array_equal(B.rids(q, k), want[q][:k])
    ctx.close()
