"""Captured operator calls after few warm-up calls: a captured call allocates
nothing, its replays write into no other object, and its operands and result
stay usable before the first replay."""
import numpy as np
import pytest

import oracle
from oracle import wahgen as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warm", [1, 2, 9])
@pytest.mark.parametrize("d", [0.002, 0.06, 0.5])
@pytest.mark.parametrize("nbits", [31 * 512, 1 << 20, (1 << 22) + 7])
def test_captured_call(nbits, d, warm):
    import torch
    import libfastlib_b200 as L
    ctx = L.Context(0)  # a fresh context: nothing of other calls in its pool
    ps = [oracle.build_runs(G.geometric_runs(50 + i, nbits, d)) for i in range(3)]
    A, B, C = (ctx.bitvector(p) for p in ps)
    outs = [ctx.empty(A.nwords() + B.nwords()) for _ in range(4)]
    for _ in range(warm):
        for op in range(4):
            A.binop_into(op, B, outs[op])
    refs = [oracle.binop(op, ps[0], ps[1]) for op in range(4)]
    for r, (_, cnt) in zip(outs, refs):
        assert r.cnt() == cnt
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        for op in range(4):
            A.binop_into(op, B, outs[op])
        ctx.set_stream(None)
    # operands and results of the captured calls serve others before a replay
    for x, xs in ((A, ps[0]), (outs[1], refs[1][0])):
        got, want = x._binop(L.MINUS, C, False), oracle.binop(3, xs, ps[2])
        assert got.cnt() == want[1] and np.array_equal(got.write(), want[0])
    others = [ctx.bitvector(p) for p in ps for _ in range(4)]  # take what the pool holds
    ctx.sync()
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        for r, (words, cnt) in zip(outs, refs):
            assert r.cnt() == cnt and np.array_equal(r.write(), words)
    for i, o in enumerate(others):
        assert np.array_equal(o.write(), ps[i // 4])
    # and the operands again, larger calls of the context in between
    big = [oracle.build_runs(G.geometric_runs(60 + i, 4 * nbits, 0.3)) for i in range(2)]
    X, Y = (ctx.bitvector(p) for p in big)
    assert np.array_equal(X._binop(L.XOR, Y, False).write(), oracle.binop(2, *big)[0])
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(outs[0].write(), refs[0][0])
    g.reset()
    for o in others + outs + [A, B, C, X, Y]:
        o.close() if hasattr(o, "close") else None
    ctx.close()
