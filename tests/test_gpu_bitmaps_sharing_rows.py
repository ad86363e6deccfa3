"""Ranges over bitmaps that are no partition of the rows: rows in several
bitmaps (every bitmap counts in whole) and rows in none (never a hit), with
cumulative rows per bitmap, at a stride and none."""
import numpy as np
import pytest

from oracle import wahgen as G

pytestmark = pytest.mark.gpu


def _serial(bits):
    """A bitmap's literal words, a run of all-ones groups as one fill."""
    n = len(bits) // 31
    words = []
    for g in bits[:31 * n].reshape(n, 31):
        w = int("".join("1" if b else "0" for b in g), 2)
        if w == 0x7FFFFFFF and words and words[-1] >= 0xC0000000:
            words[-1] += 1
        else:
            words.append(0xC0000001 if w == 0x7FFFFFFF else w)
    tail = bits[31 * n:]
    return G.serialize(words, len(tail), int("".join("1" if b else "0" for b in tail) or "0", 2))


def _index(L, ctx, sets):
    ser = [np.asarray(_serial(s), np.uint32) for s in sets]
    offs = np.concatenate([[0], np.cumsum([len(s) for s in ser])]).astype(np.int64)
    return L.Index(ctx, L.RELIC, len(sets[0]), np.arange(1.0, len(sets) + 1), offs, np.concatenate(ser))


def _check(L, ctx, idx, sets, spans):
    want = [np.flatnonzero(np.any(sets[a:b], axis=0)) for a, b in spans]
    terms = [[idx.term(a + 1.0, b + 1.0)] for a, b in spans]
    B = L.Batch(ctx, terms)
    B.run()
    assert B.counts().tolist() == [len(w) for w in want]
    for t, w in zip(terms, want):
        n, ids, hits = L.evaluate(ctx, t, want_hits=True)
        assert n == len(w) and np.array_equal(ids, w) and np.array_equal(hits.rids(), w)
        assert np.array_equal(L.evaluate(ctx, t)[1], w)


@pytest.mark.parametrize("stride", [0, 1, 2, 8])
@pytest.mark.parametrize("rows", [62, 31 * 4096 + 5])
@pytest.mark.parametrize("kind", ["equal", "some", "gaps", "last"])
def test_ranges(gpu_ctx, kind, rows, stride):
    import libfastlib_b200 as L
    rng = np.random.default_rng(rows + stride)
    n = 2 if kind == "equal" else 19
    if kind == "equal":  # the same rows twice
        sets = np.repeat(rng.random((1, rows)) < 0.5, 2, axis=0)
        sets[:, :31] = True
    else:
        owner = rng.integers(0, n + (1 if kind == "gaps" else 0), rows)
        sets = np.stack([owner == j for j in range(n)])
        if kind == "some":
            sets |= rng.random((n, rows)) < 0.02
        elif kind == "last":  # only the last bitmap shares a row
            sets[-1, np.flatnonzero(owner == 3)[:1]] = True
    old = gpu_ctx.get_tuning(L.TUNE_CUM_STRIDE)
    gpu_ctx.set_tuning(L.TUNE_CUM_STRIDE, stride)
    try:
        idx = _index(L, gpu_ctx, sets)
    finally:
        gpu_ctx.set_tuning(L.TUNE_CUM_STRIDE, old)
    spans = [(0, n), (1, n), (0, n - 1), (n - 1, n)] + [tuple(sorted(rng.choice(n + 1, 2, replace=False))) for _ in range(6)]
    _check(L, gpu_ctx, idx, sets, spans)
    idx.close()
