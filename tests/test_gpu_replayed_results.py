"""A result that a captured call writes changes with every replay: neither the
row index that an ordinary call left with it nor metadata read along with
another result's before the replay may serve its words afterwards."""
import numpy as np
import pytest

import oracle
from oracle import wahgen as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [0, 4])
@pytest.mark.parametrize("d", [0.002, 0.06, 0.5])
@pytest.mark.parametrize("nbits", [31 * 512, (1 << 22) + 7])
def test_replay_over_an_ordinary_result(nbits, d, engine):
    import torch
    import libfastlib_b200 as L
    ctx = L.Context(0)
    ctx.set_tuning(L.TUNE_DENSE_ENGINE, engine)
    px, py, pz = (oracle.build_runs(G.geometric_runs(70 + i, nbits, d)) for i in range(3))
    X, Y, Z = (ctx.bitvector(p) for p in (px, py, pz))
    out, other = (ctx.empty(X.nwords() + Y.nwords()) for _ in range(2))
    both, either = oracle.binop(0, px, py), oracle.binop(1, px, py)
    want = oracle.binop(3, both[0], pz)
    # past the first calls of a context
    for _ in range(10):
        X.binop_into(L.OR, Y, out)
        X.binop_into(L.AND, Y, other)
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        X.binop_into(L.AND, Y, out)
        ctx.set_stream(None)
    for _ in range(2):
        X.binop_into(L.OR, Y, out)
        X.binop_into(L.XOR, Y, other)
        assert other.cnt() == oracle.binop(2, px, py)[1]  # not out's metadata: they are those of OR
        ctx.sync()
        g.replay()
        torch.cuda.synchronize()
        assert out.cnt() == both[1] and np.array_equal(out.write(), both[0])
        for _ in range(2):
            got = out._binop(L.MINUS, Z, False)
            assert got.cnt() == want[1] and np.array_equal(got.write(), want[0])
    # and an ordinary call's own words again
    X.binop_into(L.OR, Y, out)
    got, ref = out._binop(L.AND, Z, False), oracle.binop(0, either[0], pz)
    assert got.cnt() == ref[1] and np.array_equal(got.write(), ref[0])
    g.reset()
    ctx.close()
