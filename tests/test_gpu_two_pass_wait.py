"""A tile of the two-pass kernels that gives up its wait for its words (made by
WAHGPU_TEST_WITHHOLD_TILE): the call reports WAHGPU_ETIMEOUT, nothing is
written by the counts of tiles that gave up, and the next call is exact."""
import numpy as np
import pytest

import oracle
from oracle import wahgen as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [0, 1, 70, -1])
def test_a_tile_that_gives_up(tile):
    import libfastlib_b200 as L
    ctx = L.Context(0)
    nbits = 31 * (512 * 101 + 7)  # 102 tiles
    a, b = (oracle.build_runs(G.geometric_runs(51 + i, nbits, 0.4)) for i in range(2))
    A, B = ctx.bitvector(a), ctx.bitvector(b)
    refs = [oracle.binop(op, a, b) for op in range(4)]
    for op in range(4):  # counts of other results are left in the scratch
        assert A._binop(op, B, False).cnt() == refs[op][1]
    ctx.set_tuning(L.TEST_WITHHOLD_TILE, tile if tile >= 0 else 101)
    r = A._binop(L.XOR, B, False)
    with pytest.raises(L.WahError) as e:
        r.write()
    assert e.value.code == -7  # WAHGPU_ETIMEOUT
    for op in range(4):
        r = A._binop(op, B, False)
        assert np.array_equal(r.write(), refs[op][0]) and r.cnt() == refs[op][1]
    ctx.close()
