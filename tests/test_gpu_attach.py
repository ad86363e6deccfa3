"""Attaching an index: the chunked passes over its words (chunk edges, words
that span tiles, list words of 32 bitmaps) against a scan of the column."""
import numpy as np
import pytest

from libfastlib_b200 import workloads as W

pytestmark = pytest.mark.gpu

TILE = 4096 * 31  # rows of one range tile


def _triple(vals, card):
    """Keys, offsets and serialized bitmaps of a relic index of `vals`."""
    n = len(vals)
    G, anb = n // 31, n % 31
    words, offs = [], [0]
    w = 1 << np.arange(30, -1, -1)
    for v in range(card):
        bits = vals == v
        groups = (bits[:31 * G].reshape(G, 31) * w).sum(1).astype(np.uint32)
        aval = 0
        for b in bits[31 * G:]:
            aval = aval << 1 | int(b)
        s = W.canonical_wah(groups, anb, aval)
        words.append(s)
        offs.append(offs[-1] + len(s))
    return np.arange(card, dtype=np.float64), np.asarray(offs, np.int64), np.concatenate(words)


def _columns():
    rng = np.random.default_rng(8)
    for n, card in [(1, 1), (31, 2), (62, 3), (31 * 511, 2), (31 * 512 + 5, 2), (31 * 513, 3), (TILE - 1, 31),
                    (TILE, 32), (TILE + 31, 33), (2 * TILE + 17, 70)]:
        yield f"mixed-{n}-{card}", rng.integers(0, card, n), card
        # sorted and run-sorted: 1-fills over chunk and tile boundaries
        yield f"sorted-{n}-{card}", np.sort(rng.integers(0, card, n)), card
        yield f"runs-{n}-{card}", np.repeat(rng.integers(0, card, n // 700 + 1), 700)[:n], card


@pytest.mark.parametrize("stride", [0, 1, 8])  # cumulative rows: auto, none, every 8 bitmaps
@pytest.mark.parametrize("name,vals,card", [pytest.param(*c, id=c[0]) for c in _columns()])
def test_attached_index_answers(gpu_ctx, name, vals, card, stride):
    import libfastlib_b200 as L
    old = gpu_ctx.get_tuning(L.TUNE_CUM_STRIDE)
    gpu_ctx.set_tuning(L.TUNE_CUM_STRIDE, stride)
    try:
        idx = L.Index(gpu_ctx, L.RELIC, len(vals), *_triple(vals, card))
    finally:
        gpu_ctx.set_tuning(L.TUNE_CUM_STRIDE, old)
    spans = [(0, card), (0, max(1, card - 1)), (card // 2, card), (1, max(2, card - 1))]
    spans += [(v, v + 1) for v in {0, card // 3, card - 1}]
    for lo, hi in spans:
        n, rids, _ = L.evaluate(gpu_ctx, [idx.term(lo, hi)])
        want = np.flatnonzero((vals >= lo) & (vals < hi))
        assert n == len(want) and np.array_equal(rids, want), (lo, hi)
    assert L.estimate_count(gpu_ctx, idx.term(0, card)) == len(vals)
    idx.close()


@pytest.mark.parametrize("bad,code", [(0x80000000, -5), (0xC0000000, -5), (0x80000000 | 600, -6)])
def test_attach_refuses_bad_words(gpu_ctx, bad, code):
    """A fill of length 0, and a bitmap of more bits than the column has
    rows, in a chunk after the first."""
    import libfastlib_b200 as L
    words = np.asarray([5] * 700 + [bad] + [9] * 50 + [0], np.uint32)
    with pytest.raises(L.WahError) as e:
        L.Index(gpu_ctx, L.RELIC, 31 * 800, [1.0], [0, len(words)], words)
    assert e.value.code == code
