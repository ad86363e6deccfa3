"""The group-space engine on every path that can take it: operators on the
reference's _c2 path (count-1 fills told from the words around one-group
runs), canonical results, copies and complements, and chains whose operands'
row index came with an earlier result; against the oracle, at the edges of
rows (32 groups), tiles (512) and CTAs (4096)."""
import numpy as np
import pytest

import oracle
from oracle import wahgen as G

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 31, 32, 33, 64, 511, 512, 513, 1024, 4095, 4096, 4097, 9001]


def _words(rng, ngroups, pfill, pone, plit, maxc):
    """Words over ngroups groups: fills (a share of them of one group), mixed
    literals, lone all-0 / all-1 literals, equal neighbours allowed."""
    out, g = [], 0
    while g < ngroups:
        if rng.random() < pfill:
            c = 1 if rng.random() < pone else int(rng.integers(1, maxc + 1))
            c = min(c, ngroups - g)
            out.append(G.fill(int(rng.integers(0, 2)), c))
            g += c
        else:
            out.append(int(rng.integers(1, 0x7FFFFFFF)) if rng.random() < plit else int(rng.choice([0, 0x7FFFFFFF])))
            g += 1
    return out


def _pairs(seed, ngroups, n):
    rng = np.random.default_rng(seed)
    done = 0
    while done < n:
        anb = int(rng.integers(0, 31))
        s = []
        for _ in range(2):
            w = _words(rng, ngroups, rng.random(), rng.random() * 0.7, rng.random(), int(rng.choice([3, 9, 60, 700])))
            s.append(np.asarray(G.serialize(w, anb, int(rng.integers(0, 1 << 31))), np.uint32))
        if oracle.is_degenerate(s[0]) or oracle.is_degenerate(s[1]):
            continue
        done += 1
        yield s


@pytest.mark.parametrize("ngroups", SIZES)
def test_operators(gpu_ctx, ngroups):
    for a, b in _pairs(ngroups, ngroups, 40 if ngroups < 2000 else 12):
        A, B = gpu_ctx.bitvector(a), gpu_ctx.bitvector(b)
        for ip in (False, True):
            for op in range(4):
                ref, cnt = oracle.binop(op, a, b, inplace=ip)
                # the first uses may take word space, the later ones take group space
                r = A._binop(op, B, ip)
                assert np.array_equal(r.write(), ref) and r.cnt() == cnt, (ngroups, op, ip)


@pytest.mark.parametrize("ngroups", SIZES)
def test_chains(gpu_ctx, ngroups):
    """((a | b) & c) - a and its complement: operands that are results."""
    rng = np.random.default_rng(1000 + ngroups)
    pairs = list(_pairs(2000 + ngroups, ngroups, 16))
    for k in range(0, len(pairs), 2):
        (a, b), (c, _) = pairs[k], pairs[k + 1]
        anb = a[-1]  # one size for all
        c = np.concatenate([c[:-2] if 0 < c[-1] < 31 else c[:-1], a[-2:] if 0 < anb < 31 else a[-1:]])
        A, B, C = (gpu_ctx.bitvector(x) for x in (a, b, c))
        ops = rng.integers(0, 4, 3)
        ref, dev = a, A
        for op, (o, O) in zip(ops, ((b, B), (c, C), (a, A))):
            if oracle.is_degenerate(ref) or oracle.is_degenerate(o):
                break
            ref, cnt = oracle.binop(int(op), ref, o)
            dev = dev._binop(int(op), O, False)
            assert np.array_equal(dev.write(), ref) and dev.cnt() == cnt, (ngroups, ops)
        else:
            assert np.array_equal(dev.flip().write(), oracle.compress(oracle.flip(ref))[0]), ngroups
            assert np.array_equal(dev.rids(), oracle.rids(oracle.flip(ref)))


@pytest.mark.parametrize("ngroups", SIZES)
def test_copies(gpu_ctx, ngroups):
    """compress() and flip(), count-1 fills of the operand kept."""
    for a, b in _pairs(3000 + ngroups, ngroups, 20):
        for s in (a, b):
            v = gpu_ctx.bitvector(s)
            assert np.array_equal(v.compress().write(), oracle.compress(s)[0]), ngroups
            v = gpu_ctx.bitvector(s)
            assert np.array_equal(v.flip().write(), oracle.compress(oracle.flip(s))[0]), ngroups
            v = gpu_ctx.bitvector(s)
            # one word per group is uncompressed already, whatever the words
            dense = s if v.nwords() == ngroups else oracle.decompress(s)
            v.decompress()
            assert np.array_equal(v.write(), dense), ngroups
            assert v.cnt() == len(oracle.rids(s))
            assert np.array_equal(v.compress().write(), oracle.compress(dense)[0]), ngroups


def test_long_runs(gpu_ctx):
    """Fills over many tiles and CTAs, heads far apart, results of one word."""
    ng = 300_000
    z, o = G.fill(0, ng), G.fill(1, ng)
    mid = [G.fill(0, 100_000), 5, G.fill(1, 1), G.fill(0, 99_998), G.fill(1, ng - 200_000)]
    far = [G.fill(1, 150_001), 7, G.fill(0, ng - 150_002)]
    vs = [np.asarray(G.serialize(w, 3, 5), np.uint32) for w in ([z], [o], mid, far)]
    for a in vs:
        for b in vs:
            A, B = gpu_ctx.bitvector(a), gpu_ctx.bitvector(b)
            for op in range(4):
                ref, cnt = oracle.binop(op, a, b)
                for _ in range(2):
                    r = A._binop(op, B, False)
                    assert np.array_equal(r.write(), ref) and r.cnt() == cnt
