"""Range evaluation from a cumulative row per bitmap (the default where it
fits), against a scan of the columns and beside indexes that keep fewer rows
or none: counts, counts alone (edge bins counted by themselves), row ids in
every order, limits per query and hit bitvectors, at the edges of the tiles
(1024 and 4096 groups of 31 rows)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL, TILE = 1024 * 31, 4096 * 31


def _columns(n, seed):
    rng = np.random.default_rng(seed)
    f = np.where(rng.random(n) < 0.7, rng.normal(size=n), rng.integers(0, 9, n)).astype(np.float32)
    return {
        "u32": rng.integers(0, 40, n).astype(np.uint32),
        "i32 sorted": np.sort(rng.integers(-30, 30, n)).astype(np.int32),
        "f32 bins": f,
        "f32 clustered bins": np.sort(f),
    }


def _queries(rng, cols, nq):
    names = list(cols)
    out = []
    for _ in range(nq):
        terms = []
        for c in rng.choice(len(names), size=int(rng.integers(1, 4)), replace=False):
            v = cols[names[c]]
            lo, hi = np.sort(rng.choice(v, 2)).astype(np.float64)
            lop, rop = int(rng.integers(0, 3)), int(rng.integers(0, 3))
            terms.append((names[c], float(lo) if lop else None, float(hi) if rop else None, max(lop, 1), max(rop, 1)))
        out.append(terms)
    # nothing, everything, one value, past the ends
    k = names[0]
    out += [[(k, 7.0, 7.0, 1, 1)], [(k, None, None, 1, 1)], [(k, 5.0, 5.0, 2, 2)], [(k, 100.0, None, 1, 1)]]
    return out


def _scan(cols, q, n):
    m = np.ones(n, bool)
    for name, lo, hi, lop, rop in q:
        v = cols[name].astype(np.float64)
        if lo is not None:
            m &= (lo < v) if lop == 1 else (lo <= v)
        if hi is not None:
            m &= (v < hi) if rop == 1 else (v <= hi)
    return np.flatnonzero(m).astype(np.uint32)


@pytest.mark.parametrize("n", [1, 31, 40, SMALL - 1, SMALL, SMALL + 32, TILE - 31, TILE, TILE + 5, 3 * TILE + 77])
@pytest.mark.parametrize("strides", [(0, 0), (0, 8), (1, 0)])  # of the first two columns, of the others: auto, 8, none
def test_rows_against_scan(gpu_ctx, n, strides):
    import libfastlib_b200 as L
    cols = _columns(n, n)
    idx = {}
    try:
        for i, (name, v) in enumerate(cols.items()):
            gpu_ctx.set_tuning(L.TUNE_CUM_STRIDE, strides[i // 2])
            if "bins" in name:
                idx[name] = L.Index.build(gpu_ctx, L.BIN, v, nbins=50)
            else:
                idx[name] = L.Index.build(gpu_ctx, L.RELIC, v)
                idx[name].set_values(v)
    finally:
        gpu_ctx.set_tuning(L.TUNE_CUM_STRIDE, 0)
    rng = np.random.default_rng(n + 1)
    qs = _queries(rng, cols, 24)
    want = [_scan(cols, q, n) for q in qs]
    terms = [[idx[c].term(lo, hi, lop, rop) for c, lo, hi, lop, rop in q] for q in qs]
    counts = [len(w) for w in want]

    B = L.Batch(gpu_ctx, terms)  # counts alone
    for _ in range(2):
        B.run()
        assert B.counts().tolist() == counts
    single = [t for t in terms if len(t) == 1]
    B = L.Batch(gpu_ctx, single)  # one-term queries only
    B.run()
    assert B.counts().tolist() == [c for c, t in zip(counts, terms) if len(t) == 1]

    caps = [int(rng.integers(0, 2 * max(c, 1))) for c in counts]
    for order in (1, 0, 2):
        gpu_ctx.set_tuning(L.TUNE_RANGE_ORDER, order)
        try:
            B = L.Batch(gpu_ctx, terms, rid_cap=max(sum(counts), 1))
            B.run()
            assert B.counts().tolist() == counts, order
            for q, w in enumerate(want):
                assert np.array_equal(B.rids(q, len(w)), w), (order, q)
            B = L.Batch(gpu_ctx, terms, caps=caps)
            B.run()
            assert B.counts().tolist() == counts, order
            for q, w in enumerate(want):
                if sum(caps):
                    assert np.array_equal(B.rids(q, min(caps[q], len(w))), w[:caps[q]]), (order, q)
        finally:
            gpu_ctx.set_tuning(L.TUNE_RANGE_ORDER, 1)
    for q in range(0, len(qs), 5):
        c, rids, hits = L.evaluate(gpu_ctx, terms[q], want_hits=True)
        assert c == counts[q] and np.array_equal(rids, want[q])
        assert hits.size() == n and np.array_equal(hits.rids(), want[q])
    for i in idx.values():
        i.close()


def test_overlapping_bitmaps_are_not_added_up(gpu_ctx):
    """Bitmaps that share rows (no equality encoding): a count is that of
    their OR, not the sum of theirs."""
    import libfastlib_b200 as L
    one = np.asarray([0x7FFFFFFF, 0x00000003, 0], np.uint32)
    idx = L.Index(gpu_ctx, L.RELIC, 62, [1.0, 2.0], [0, 3, 6], np.concatenate([one, one]))
    B = L.Batch(gpu_ctx, [[idx.term(1.0, 3.0)]])
    B.run()
    assert B.counts().tolist() == [33]
    assert L.estimate_count(gpu_ctx, idx.term(1.0, 3.0)) == 66
    idx.close()
