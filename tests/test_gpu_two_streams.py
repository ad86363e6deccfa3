"""A result launched before its context was given another stream: its metadata
wait for the stream it was launched on."""
import numpy as np
import pytest

import oracle
from oracle import wahgen as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [0.002, 0.5])
def test_result_of_another_stream(d):
    import torch
    import libfastlib_b200 as L
    ctx = L.Context(0)
    pa, pb = (oracle.build_runs(G.geometric_runs(90 + i, 1 << 20, d)) for i in range(2))
    A, B = ctx.bitvector(pa), ctx.bitvector(pb)
    for op in range(4):  # what the calls allocate is there
        assert A._binop(op, B, False).cnt() == oracle.binop(op, pa, pb)[1]
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(2):
        ctx.set_stream(s1.cuda_stream)
        with torch.cuda.stream(s1):
            torch.cuda._sleep(40_000_000)  # some 20 ms ahead of the operators
        first = A._binop(L.AND, B, False)
        along = A._binop(L.XOR, B, False)
        ctx.set_stream(s2.cuda_stream)
        second = first._binop(L.MINUS, A, False)  # its operand was launched on s1
        third = A._binop(L.OR, B, False)
        words, cnt = oracle.binop(0, pa, pb)
        for r, (ref, c) in ((along, oracle.binop(2, pa, pb)), (third, oracle.binop(1, pa, pb)), (first, (words, cnt)),
                            (second, oracle.binop(3, words, pa))):
            assert r.cnt() == c and np.array_equal(r.write(), ref)
        torch.cuda.synchronize()
    ctx.set_stream(None)
    ctx.close()
