"""Metadata of several results read together: whatever is asked for first,
freed in between or launched on another stream, and results whose launch was
only captured."""
import numpy as np
import pytest

import oracle
from oracle import wahgen as G

pytestmark = pytest.mark.gpu


def _pairs(n):
    out = []
    for i in range(n):
        d = 0.002 * (1 + i % 60)
        out.append(tuple(oracle.build_runs(G.geometric_runs(100 + 2 * i + k, 31 * (40 + 13 * (i % 9)) + i % 31, d))
                         for k in (0, 1)))
    return out


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 300])
def test_many_results(gpu_ctx, n):
    rng = np.random.default_rng(n)
    ps = _pairs(n)
    res = []
    for i, (a, b) in enumerate(ps):
        r = gpu_ctx.bitvector(a)._binop(i % 4, gpu_ctx.bitvector(b), False)
        res.append(r if rng.random() < 0.8 else None)  # some results are dropped unread
    for i in rng.permutation(n):
        if res[i] is None:
            continue
        ref, cnt = oracle.binop(int(i) % 4, *ps[i])
        assert res[i].cnt() == cnt and res[i].nwords() == len(ref) - (2 if 0 < ref[-1] < 31 else 1)
        assert np.array_equal(res[i].write(), ref)
        if rng.random() < 0.3:
            res[i] = None


def test_captured_result_is_read_after_its_replay(gpu_ctx):
    import torch
    import libfastlib_b200 as L
    (a, b), (c, d) = _pairs(2)
    A, B = gpu_ctx.bitvector(a), gpu_ctx.bitvector(b)
    out = gpu_ctx.empty(A.nwords() + B.nwords())
    A.binop_into(L.OR, B, out)  # allocates what the launches need
    assert out.cnt() == oracle.binop(1, a, b)[1]
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        gpu_ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        A.binop_into(L.AND, B, out)
        gpu_ctx.set_stream(None)
    # another result's metadata are read before the graph runs
    C = gpu_ctx.bitvector(c)._binop(L.XOR, gpu_ctx.bitvector(d), False)
    assert C.cnt() == oracle.binop(2, c, d)[1]
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    ref, cnt = oracle.binop(0, a, b)
    assert out.cnt() == cnt and np.array_equal(out.write(), ref)
