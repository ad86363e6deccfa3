"""Two-pass results whose heads lie far apart: the run of a head ends at the
next one, found in the tiles after it, in the rest of a CTA's range or by the
warps' first heads beyond."""
import numpy as np
import pytest

import oracle
from oracle import wahgen as G

pytestmark = pytest.mark.gpu
T = 512  # groups per tile


def _islands(groups, at, one):
    """Runs of `one` groups but for literals at the groups given."""
    words, p, h = [], 0, 0xC0000000 if one else 0x80000000
    for g in sorted(set(at)):
        if g > p:
            words.append(h | (g - p) if g - p > 1 else (0x7FFFFFFF if one else 0))
        words.append(0x2AAAAAAA)
        p = g + 1
    if groups > p:
        words.append(h | (groups - p) if groups - p > 1 else (0x7FFFFFFF if one else 0))
    return np.asarray(G.serialize(words, 3, 5), np.uint32)


@pytest.mark.parametrize("tiles", [33, 34, 300, 3000, 5003])
def test_heads_far_apart(gpu_ctx, tiles):
    import libfastlib_b200 as L
    groups = tiles * T - 3
    dense = oracle.build_runs(G.geometric_runs(tiles, 31 * groups + 3, 0.5))
    A, B = gpu_ctx.bitvector(dense), gpu_ctx.bitvector(dense)
    last = groups - 1
    spots = [[], [0], [last], [0, last], [T - 1, T], [33 * T - 1 if tiles > 33 else 5, last],
             [tiles // 2 * T], [tiles // 3 * T + 7, tiles // 2 * T - 1, last - T],
             list(range(0, groups, 97 * T)), list(range(T - 1, groups, 41 * T))]
    for one in (False, True):
        for at in spots:
            p = _islands(groups, at, one)
            P = gpu_ctx.bitvector(p)
            for op in (L.OR, L.MINUS) if one else (L.AND, L.XOR):
                r, (ref, cnt) = A._binop(op, P, False), oracle.binop(op, dense, p)
                assert r.cnt() == cnt and np.array_equal(r.write(), ref), (one, at, op)
                # the result's row index serves the next operator
                r2, (ref2, cnt2) = r._binop(L.XOR, A, False), oracle.binop(2, ref, dense)
                assert r2.cnt() == cnt2 and np.array_equal(r2.write(), ref2), (one, at, op)
    r = A._binop(L.XOR, B, False)
    ref, cnt = oracle.binop(2, dense, dense)
    assert cnt == 0 and r.cnt() == 0 and np.array_equal(r.write(), ref)
