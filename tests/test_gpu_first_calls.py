"""A context's calls do the same work from the second one on: the engine of an
operator, and whether its result keeps a row index, do not depend on how many
calls there have been."""
import numpy as np
import pytest

import oracle
from oracle import wahgen as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [0.06, 0.5])
def test_launches_per_call(d):
    import libfastlib_b200 as L
    ctx = L.Context(0)
    pa, pb = (oracle.build_runs(G.geometric_runs(30 + i, 1 << 24, d)) for i in range(2))
    A, B = ctx.bitvector(pa), ctx.bitvector(pb)
    either = oracle.binop(1, pa, pb)
    ref, cnt = oracle.binop(2, either[0], pa)
    out, out2 = ctx.empty(A.nwords() + B.nwords()), ctx.empty(2 * (A.nwords() + B.nwords()))
    per = []
    for _ in range(12):
        l0 = ctx.launches
        A.binop_into(L.OR, B, out)
        l1 = ctx.launches
        out.binop_into(L.XOR, A, out2)
        per.append((l1 - l0, ctx.launches - l1))
        assert out2.cnt() == cnt
    assert np.array_equal(out2.write(), ref)
    # the operands' row indexes are made in the first call
    assert per[0] == (4, 2) and set(per[1:]) == {(2, 2)}, per
    ctx.close()
