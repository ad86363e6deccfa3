"""Captured calls keep the look-back scratch they were captured with: later
calls of the context may need more of it, and get another block."""
import numpy as np
import pytest

from oracle import wahgen as G

pytestmark = pytest.mark.gpu


def _literals(seed, n):
    """n words: a 0-fill of two groups, the others literals, none uniform."""
    w = np.random.default_rng(seed).integers(1, 0x7FFFFFFF, n, dtype=np.uint32)
    w[0] = 0x80000002
    return np.concatenate([w, np.asarray(G.serialize([], 3, 5), np.uint32)])


def _bits(words):
    return int(np.bitwise_count(words[1:]).sum())


def test_replays_after_the_scratch_has_grown():
    import torch
    import libfastlib_b200 as L
    ctx = L.Context(0)
    rng = np.random.default_rng(3)
    n = 1_000_003
    cols = [rng.integers(0, 50, n).astype(np.uint32) for _ in range(2)]
    idx = [L.Index.build(ctx, L.RELIC, c) for c in cols]
    spans = [[tuple(sorted(rng.choice(51, 2, replace=False))) for _ in range(2)] for _ in range(400)]
    # conjunctions, so that their 9 x 400 items are claimed from the scratch
    B = L.Batch(ctx, [[x.term(float(a), float(b)) for x, (a, b) in zip(idx, s)] for s in spans])
    B.run()
    want = B.counts()
    for s, c in list(zip(spans, want))[::40]:
        assert c == np.count_nonzero(np.logical_and(*[(v >= a) & (v < b) for v, (a, b) in zip(cols, s)]))
    ctx.set_tuning(L.TUNE_DENSE_ENGINE, 2)  # operators through the merge
    pa, pb = _literals(1, 5000), _literals(2, 5000)
    X, Y = ctx.bitvector(pa), ctx.bitvector(pb)
    out = ctx.empty(X.nwords() + Y.nwords())
    X.binop_into(L.AND, Y, out)
    both = out.write()
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        B.run()
        X.binop_into(L.AND, Y, out)
        ctx.set_stream(None)
    torch.cuda.synchronize()
    for words in (1 << 21, 1 << 22):  # row ids of 1024 words a tile, more tiles than the block holds
        big = _literals(4, words)
        V = ctx.bitvector(big)
        assert len(V.rids()) == _bits(big[:words]) + 2
        for _ in range(3):
            X.binop_into(L.OR, Y, out)
            B.run()  # its counts are read after the replay
            ctx.sync()
            g.replay()
            torch.cuda.synchronize()
            assert np.array_equal(B.counts(), want)
            assert np.array_equal(out.write(), both)
    g.reset()
    ctx.close()


def test_a_captured_call_does_not_grow_the_scratch():
    import torch
    import libfastlib_b200 as L
    ctx = L.Context(0)
    ctx.set_tuning(L.TUNE_DENSE_ENGINE, 2)
    ctx.set_tuning(L.TUNE_MERGE_TILE, 16)
    pa, pb = _literals(5, 400_000), _literals(6, 400_000)  # 1563 tiles of the merge, 98 of the upload
    X, Y = ctx.bitvector(pa), ctx.bitvector(pb)
    out = ctx.empty(X.nwords() + Y.nwords())
    assert X.nwords() == Y.nwords() == 400_000
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        with pytest.raises(L.WahError) as e:
            X.binop_into(L.AND, Y, out)
        ctx.set_stream(None)
    assert e.value.code == -3  # WAHGPU_ECUDA
    X.binop_into(L.AND, Y, out)  # the call itself is as good as before
    w = pa[:400_000] & pb[:400_000]
    assert out.cnt() == _bits(w) + 2
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        X.binop_into(L.AND, Y, out)
        ctx.set_stream(None)
    g.replay()
    torch.cuda.synchronize()
    assert out.cnt() == _bits(w) + 2
    g.reset()
    ctx.close()
