"""A merge tile that publishes only after a wait for it has given up (made on
the device by WAHGPU_TEST_WITHHOLD_TILE, every wait bounded): the call reports
WAHGPU_ETIMEOUT whichever tile it is, the first one too, and the next call is
exact."""
import numpy as np
import pytest

import oracle
from oracle import wahgen as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [0, 1])
def test_late_tile(tile):
    import libfastlib_b200 as L
    ctx = L.Context(0)
    ctx.set_tuning(L.TUNE_MERGE_TILE, 16)  # operators through the merge
    a, b = (oracle.build_runs(G.geometric_runs(41 + i, 1 << 21, 0.002)) for i in range(2))
    A, B = ctx.bitvector(a), ctx.bitvector(b)
    assert A.nwords() + B.nwords() > 3 * 16 * 32  # some tiles
    ref, cnt = oracle.binop(1, a, b)
    assert A._binop(L.OR, B, False).cnt() == cnt
    ctx.set_tuning(L.TEST_WITHHOLD_TILE, tile)
    with pytest.raises(L.WahError) as e:
        A._binop(L.OR, B, False).write()
    assert e.value.code == -7  # WAHGPU_ETIMEOUT
    for _ in range(2):
        r = A._binop(L.OR, B, False)
        assert np.array_equal(r.write(), ref) and r.cnt() == cnt
    ctx.close()
