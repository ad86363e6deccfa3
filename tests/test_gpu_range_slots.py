"""Row ids of two-pass batches around the number of hits per tile that the
count pass keeps (32): in one warp's rows or all over the tile, with limits
inside, at and past them, against a scan."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE = 4096 * 31


@pytest.mark.parametrize("stride", [0, 8])
@pytest.mark.parametrize("n", [TILE // 4, 3 * TILE + 17])
def test_ids_of_few_hits(gpu_ctx, n, stride):
    import libfastlib_b200 as L
    rng = np.random.default_rng(n + stride)
    v = np.full(n, 99, dtype=np.uint32)
    per_tile = (0, 1, 2, 31, 32, 33, 64)
    for t0 in range(0, n, TILE):
        rows = rng.permutation(np.arange(t0, min(t0 + TILE, n)))
        at = 0
        for k, c in enumerate(per_tile):
            c = min(c, len(rows) - at)
            v[rows[at:at + c]] = 10 + k  # scattered
            at += c
    # and close together: the first rows of the second tile, or of the only one
    s = TILE if n > TILE else 0
    for k, c in enumerate(per_tile):
        v[s + 100 * k:s + 100 * k + c] = 30 + k
    gpu_ctx.set_tuning(L.TUNE_CUM_STRIDE, stride)
    gpu_ctx.set_tuning(L.TUNE_RANGE_ORDER, 2)
    try:
        ix = L.Index.build(gpu_ctx, L.RELIC, v)
        ranges = [(float(a), float(a + w)) for a in (10, 11, 13, 14, 15, 16, 30, 31, 33, 34, 35, 36) for w in (1, 2, 8)]
        want = [np.flatnonzero((v >= lo) & (v < hi)) for lo, hi in ranges]
        terms = [[ix.term(lo, hi)] for lo, hi in ranges]
        B = L.Batch(gpu_ctx, terms, rid_cap=sum(map(len, want)))
        B.run()
        assert B.counts().tolist() == [len(w) for w in want]
        for q, w in enumerate(want):
            assert np.array_equal(B.rids(q, len(w)), w), q
        for caps in ([1 + 31 * (q % 4) for q in range(len(want))], [len(w) for w in want], [10_000] * len(want)):
            B = L.Batch(gpu_ctx, terms, caps=caps)
            for _ in range(2):
                B.run()
                assert B.counts().tolist() == [len(w) for w in want]
                for q, w in enumerate(want):
                    assert np.array_equal(B.rids(q, min(caps[q], len(w))), w[:caps[q]]), q
        ix.close()
    finally:
        gpu_ctx.set_tuning(L.TUNE_CUM_STRIDE, 0)
        gpu_ctx.set_tuning(L.TUNE_RANGE_ORDER, 1)
