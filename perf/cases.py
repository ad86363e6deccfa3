"""Performance cases: the work a program has this library do, through its
public entry points, with the inputs such a program holds on the GPU.

Every output is a whole number (WAH words, row ids, counts), so results are
compared bit for bit and no case has a value "in 64 bits".  Buffers that hold
a result of varying length are sized by the case, zero past its end.
"""
import ctypes
import math

import numpy as np
import torch

import libfastlib_b200 as L
from libfastlib_b200 import workloads as W

ALLONES = 0x7FFFFFFF
MEAN1 = 8.0  # mean length of the 1-runs of the raw bit patterns
OPS = (L.AND, L.OR, L.XOR, L.MINUS)
NAMES = ("and", "or", "xor", "minus")


# ------------------------------------------------------------------- cases
def listed():
    return [
        # interactive use on one table of a million rows: two predicates'
        # hit vectors combined by each operator, every result read back
        {"name": "ops_1m_rows", "kind": "ops_host", "nbits": 1_000_003, "da": 0.01, "db": 0.02},
        # the raw bitvector logic at its full 2^28 bits, from very sparse
        # predicates to incompressible ones, results kept on the device
        {"name": "ops_1e-3", "kind": "ops", "nbits": 1 << 28, "da": 1e-3, "db": 1e-3},
        {"name": "ops_1e-2", "kind": "ops", "nbits": 1 << 28, "da": 1e-2, "db": 1e-2},
        {"name": "ops_0.1", "kind": "ops", "nbits": 1 << 28, "da": 0.1, "db": 0.1},
        {"name": "ops_0.5", "kind": "ops", "nbits": 1 << 28, "da": 0.5, "db": 0.5},
        # a selective predicate against an incompressible one, ragged size
        {"name": "ops_mixed", "kind": "ops", "nbits": 99_999_989, "da": 1e-3, "db": 0.5},
        # a WHERE tree over four predicates, its row ids left on the device
        {"name": "where_rids", "kind": "where", "nbits": 50_000_017, "da": 0.02, "db": 0.03, "dc": 0.1, "dd": 0.05},
        # encode and decode: serialized words taken in, complemented,
        # expanded to one literal per group and compressed again
        {"name": "convert", "kind": "convert", "nbits": 1 << 27, "da": 0.05},
        # single range queries as they come in, count and row ids to the host
        {"name": "relic_query", "kind": "query", "rows": 1_000_000, "card": 100, "queries": 8},
        # a column that has just been loaded: its index is built, then a
        # batch of ranges answered with all row ids
        {"name": "relic_build_batch", "kind": "build", "rows": 1_000_000, "card": 100, "queries": 100},
        # a batch of binned ranges, both ends inside edge bins, counts only
        {"name": "range_batch", "kind": "range", "rows": 10_000_000, "bins": 1000, "queries": 1000},
        # a batch of 1- to 4-term conjunctions over columns of several kinds,
        # the first row ids of each query (what the query server runs)
        {"name": "conj_batch", "kind": "conj", "rows": 10_000_000, "queries": 1024, "cap": 256},
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["ops_host", "ops", "ops", "ops", "where", "convert", "query", "build", "range", "conj"])
    if kind == "ops_host":
        return {"kind": kind, "nbits": int(log(1 << 10, 1 << 22)), "da": log(1e-4, 0.5), "db": log(1e-4, 0.5)}
    if kind == "ops":
        return {"kind": kind, "nbits": int(log(1 << 18, 1 << 28)), "da": log(1e-4, 0.5), "db": log(1e-4, 0.5)}
    if kind == "where":
        return {"kind": kind, "nbits": int(log(1 << 18, 1 << 27)), "da": log(1e-3, 0.2), "db": log(1e-3, 0.2),
                "dc": log(1e-3, 0.2), "dd": log(1e-3, 0.5)}
    if kind == "convert":
        return {"kind": kind, "nbits": int(log(1 << 18, 1 << 28)), "da": log(1e-4, 0.5)}
    if kind == "query":
        return {"kind": kind, "rows": int(log(1 << 14, 1 << 22)), "card": int(log(10, 2000)), "queries": rng.randint(1, 12)}
    if kind == "build":
        return {"kind": kind, "rows": int(log(1 << 14, 1 << 22)), "card": int(log(10, 2000)), "queries": rng.randint(1, 200)}
    if kind == "range":
        return {"kind": kind, "rows": int(log(1 << 17, 10_000_000)), "bins": int(log(64, 1500)), "queries": int(log(1, 1000))}
    return {"kind": kind, "rows": int(log(1 << 17, 10_000_000)), "queries": int(log(1, 1024)), "cap": int(log(16, 2048))}


# ------------------------------------------------------------------- inputs
def _serial(seed, nbits, density):
    """Serialized WAH words (a CUDA tensor) of alternating geometric runs, a
    0-run first: 1-runs of mean MEAN1, 0-runs of mean MEAN1 (1 - d) / d."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    p0 = 1.0 / max(MEAN1 * (1.0 - density) / density, 1.0)
    ends, total = [], 0
    while total < nbits:
        n = int(1.05 * (nbits - total) / (1.0 / p0 + MEAN1)) + 512
        u = torch.rand((n, 2), generator=g, device="cuda", dtype=torch.float64)
        den = torch.tensor([math.log1p(-p0) if p0 < 1.0 else -1e30, math.log1p(-1.0 / MEAN1)], device="cuda",
                           dtype=torch.float64)
        e = torch.cumsum((torch.floor(torch.log1p(-u) / den) + 1.0).to(torch.int64).reshape(-1), 0) + total
        ends.append(e)
        total = int(e[-1])
        del u
    ends = torch.cat(ends)
    ends = ends[ends < nbits]
    mark = torch.zeros(nbits, dtype=torch.int8, device="cuda")
    mark[ends] = 1
    bits = torch.cumsum(mark, 0, dtype=torch.int32).bitwise_and_(1)
    del mark, ends
    ng, anb = nbits // 31, nbits % 31
    groups = torch.zeros(ng, dtype=torch.int32, device="cuda")
    b = bits[:31 * ng].view(ng, 31)
    for k in range(31):
        groups |= b[:, k] << (30 - k)
    aval = 0
    for v in bits[31 * ng:].tolist():
        aval = aval << 1 | v
    del bits, b
    # one word per run of equal all-0 / all-1 groups, one per mixed group
    cls = (groups == 0).to(torch.int8) + 2 * (groups == ALLONES).to(torch.int8)
    head = torch.ones(ng, dtype=torch.bool, device="cuda")
    if ng:
        head[1:] = (cls[1:] != cls[:-1]) | (cls[1:] == 0)
    h = torch.nonzero(head).reshape(-1)
    ln = torch.diff(h, append=torch.tensor([ng], device="cuda"))
    c, w = cls[h], groups[h].to(torch.int64)
    w = torch.where((c == 1) & (ln > 1), ln + 0x80000000, w)
    w = torch.where((c == 2) & (ln > 1), ln + 0xC0000000, w)
    tail = torch.tensor([aval, anb] if anb else [0], dtype=torch.int64, device="cuda")
    return torch.cat([w, tail]).to(torch.int32)


class _Words:
    """Device words of a library object as a CUDA array; the tensor made
    from it keeps the owner (and so its context's memory) alive."""

    def __init__(self, ptr, n, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (ptr, False), "version": 2}


def _view(ptr, n, owner):
    if n == 0:
        return torch.zeros(0, dtype=torch.int32, device="cuda")
    return torch.as_tensor(_Words(int(ptr), n, owner), device="cuda")


def _room(nbits, density):
    """Words that hold any operand of this size and density."""
    return int(1.1 * _words(nbits, None, density) / 4.0) + 20_000


def _result(ctx, cap):
    """A result bitvector with room for cap words, and its whole word array
    (zero where no result word is written)."""
    bv = ctx.empty(cap)
    words = _view(ctx.lib.wahgpu_bv_device_words(bv.h), cap, bv)
    words.zero_()
    return bv, words


def _uniform(seed, rows, card):
    """Every value of [0, card) equally often, in random row order."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randperm(rows, generator=g, device="cuda").remainder_(card).to(torch.int32)


def _ranges(case):
    """The case's ranges lo <= x < hi with ends in [0, card]."""
    card, n = case["card"], case["queries"]
    r = np.random.Generator(np.random.PCG64(1000 * card + n))
    out = []
    while len(out) < n:
        lo, hi = sorted(int(v) for v in r.integers(0, card + 1, size=2))
        if lo < hi:
            out.append((float(lo), float(hi)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    ctx = L.Context(0)
    st = {"kind": kind, "ctx": ctx}
    if kind in ("ops", "ops_host"):
        a = ctx.bitvector(_serial(4 * seed, case["nbits"], case["da"]))
        b = ctx.bitvector(_serial(4 * seed + 1, case["nbits"], case["db"]))
        st.update(a=a, b=b)
        cap = max(a.nwords() + b.nwords(), _room(case["nbits"], case["da"]) + _room(case["nbits"], case["db"]))
        if kind == "ops":
            st["res"] = [_result(ctx, cap) for _ in OPS]
        else:
            st["res"] = np.zeros((len(OPS), cap + 2), dtype=np.uint32)
    elif kind == "where":
        p = [ctx.bitvector(_serial(4 * seed + i, case["nbits"], case["d" + c])) for i, c in enumerate("abcd")]
        st["p"] = p
        cap = max(p[2].cnt(), int(1.25 * case["nbits"] * case["dc"]) + 20_000)
        st["rids"] = torch.zeros(cap, dtype=torch.int32, device="cuda")
    elif kind == "convert":
        st["serial"] = _serial(4 * seed, case["nbits"], case["da"])
        cap = max(st["serial"].numel(), _room(case["nbits"], case["da"]))
        st["words"] = torch.zeros(cap, dtype=torch.int32, device="cuda")
    elif kind == "query":
        st["index"] = L.Index.build(ctx, L.RELIC, _uniform(seed, case["rows"], case["card"]))
        st["ranges"] = _ranges(case)
    elif kind == "build":
        st["column"] = _uniform(seed, case["rows"], case["card"])
        st["ranges"] = _ranges(case)
        # room for the row ids: a query's expected hits and some to spare
        share = sum(hi - lo for lo, hi in st["ranges"]) / case["card"]
        st["cap"] = min(int(share * case["rows"] * 1.05) + 4096 * case["queries"], case["rows"] * case["queries"])
    elif kind == "range":
        ix = L.Index.build(ctx, L.BIN, W.mixture_column(seed, case["rows"]), nbins=case["bins"])
        nobs = ix.nbitmaps()
        q = W.binned_range_queries(seed, ix.keys(), nobs, case["queries"], max(2, nobs // 2))
        st.update(index=ix, batch=L.Batch(ctx, [[ix.term(lo, hi)] for lo, hi in q]))
    else:
        rows = case["rows"]
        cols, metas = [], []
        for i in range(2):
            cols.append(L.Index.build(ctx, L.RELIC, W.uniform_int_column(8 * seed + i, rows, 1000)))
            metas.append({"kind": "relic", "card": 1000})
        z = W.zipf_column(8 * seed + 2, rows, 1.1, 1_000_000).to(torch.int32)
        cols.append(L.Index.build(ctx, L.RELIC, z))
        metas.append({"kind": "relic", "card": 1_000_000})
        for i in range(2):
            ix = L.Index.build(ctx, L.BIN, W.normal_column(8 * seed + 4 + i, rows), nbins=512)
            cols.append(ix)
            metas.append({"kind": "bin", "keys": ix.keys(), "nobs": ix.nbitmaps(), "max_span": 128})
        q = W.conjunctive_queries(seed, metas, case["queries"])
        st["cols"] = cols
        st["batch"] = L.Batch(ctx, [[cols[c].term(lo, hi) for c, lo, hi in t] for t in q],
                              caps=[case["cap"]] * len(q))
        rids = _view(ctx.lib.wahgpu_batch_device_rids(st["batch"].h), case["cap"] * len(q), st["batch"])
        st["rids"] = rids.view(len(q), case["cap"])
        st["slot"] = torch.arange(case["cap"], device="cuda").unsqueeze(0)
    return st


# ---------------------------------------------------------------------- run
def run(st):
    kind, ctx = st["kind"], st["ctx"]
    out = {}
    if kind == "ops":
        a, b = st["a"], st["b"]
        for op, (r, _) in zip(OPS, st["res"]):
            a.binop_into(op, b, r)
        for name, (r, words) in zip(NAMES, st["res"]):
            i = r._info()
            out[name] = [words, int(i.nwords), int(i.cnt), int(i.anb), int(i.aval)]
    elif kind == "ops_host":
        a, b = st["a"], st["b"]
        for k, r in enumerate((a & b, a | b, a ^ b, a - b)):
            w = r.write()
            st["res"][k, :len(w)] = w
            out[NAMES[k]] = [len(w), r.cnt()]
        out["words"] = st["res"].view(np.int32)
    elif kind == "where":
        a, b, c, d = st["p"]
        hits = ((a | b) & c) - d
        rids = st["rids"]
        n = ctx.check(int(ctx.lib.wahgpu_bv_rids_device(hits.h, ctypes.c_void_p(rids.data_ptr()), rids.numel())))
        ctx.sync()
        out["rids"], out["count"] = rids, n
    elif kind == "convert":
        bv = ctx.bitvector(st["serial"])
        bv.flip()
        flipped = bv.cnt()
        bv.decompress()
        dense = bv.nwords()
        bv.compress()
        n = bv.nwords()
        st["words"][:n].copy_(_view(ctx.lib.wahgpu_bv_device_words(bv.h), n, bv))
        out["words"], out["counts"] = st["words"], [n, flipped, dense, bv.cnt()]
    elif kind == "query":
        ix = st["index"]
        for k, (lo, hi) in enumerate(st["ranges"]):
            n, rids, _ = L.evaluate(ctx, [ix.term(lo, hi)])
            out["q%02d" % k] = [n, rids.view(np.int32)]
    elif kind == "build":
        ix = L.Index.build(ctx, L.RELIC, st["column"])
        batch = L.Batch(ctx, [[ix.term(lo, hi)] for lo, hi in st["ranges"]], rid_cap=st["cap"])
        batch.run()
        counts = batch.counts()
        st["kept"] = (ix, batch)
        out["keys"], out["counts"] = ix.keys().astype(np.int64), counts.astype(np.int64)
        out["rids"] = _view(ctx.lib.wahgpu_batch_device_rids(batch.h), int(counts.sum()), batch)
    elif kind == "range":
        st["batch"].run()
        out["counts"] = st["batch"].counts().astype(np.int64)
    else:
        st["batch"].run()
        counts = st["batch"].counts().astype(np.int64)
        out["counts"] = counts
        # every query's ids, the slots it does not fill blank
        kept = torch.from_numpy(counts).to("cuda").unsqueeze(1)
        out["rids"] = torch.where(st["slot"] < kept, st["rids"], -1)
    return out


# --------------------------------------------------------------------- work
def _words_per_group(op, da, db):
    """Expected words per 31-bit group of (a op b) for independent run
    patterns: one per mixed group and one per run of uniform groups, so
    1 - P(two neighbouring groups all 0) - P(both all 1)."""
    def chain(d):
        p01, p10 = d / (MEAN1 * (1.0 - d)), 1.0 / MEAN1
        return np.array([1.0 - d, d]), np.array([[1.0 - p01, p01], [p10, 1.0 - p10]])

    (va, ta), (vb, tb) = chain(da), chain(db)
    v, t = np.kron(va, vb), np.kron(ta, tb)
    bit = {None: [0, 0, 1, 1], L.AND: [0, 0, 0, 1], L.OR: [0, 1, 1, 1], L.XOR: [0, 1, 1, 0], L.MINUS: [0, 0, 1, 0]}[op]
    w = 1.0
    for val in (0, 1):
        keep = np.array([1.0 if b == val else 0.0 for b in bit])
        tk = t * keep[None, :]
        w -= float((v * keep) @ np.linalg.matrix_power(tk, 61) @ np.ones(4))
    return max(w, 0.0)


def _words(nbits, op, da, db=0.5):
    return 4.0 * (nbits // 31) * _words_per_group(op, da, db) + 8.0


def _bitmap_bytes(rows, density):
    """Bytes of a bitmap of independent bits."""
    return 4.0 * (rows / 31.0) * (1.0 - (1.0 - density) ** 62)


def work(case):
    kind = case["kind"]
    if kind in ("ops", "ops_host"):
        n, da, db = case["nbits"], case["da"], case["db"]
        b = _words(n, None, da) + _words(n, None, db) + sum(_words(n, op, da, db) for op in OPS)
        return {"bytes": b, "flops": 0}
    if kind == "where":
        n = case["nbits"]
        dab = case["da"] + case["db"] - case["da"] * case["db"]
        hits = n * dab * case["dc"] * (1.0 - case["dd"])
        return {"bytes": sum(_words(n, None, case["d" + c]) for c in "abcd") + 4.0 * hits, "flops": 0}
    if kind == "convert":
        n = case["nbits"]
        # in and out compressed, and the expanded form between them
        return {"bytes": 2.0 * _words(n, None, case["da"]) + 4.0 * (n // 31), "flops": 0}
    if kind in ("query", "build"):
        # a third of the column's values on average, the smaller side read
        rows, card, nq = case["rows"], case["card"], case["queries"]
        ids = 4.0 * nq * rows / 3.0
        if kind == "build":
            return {"bytes": 4.0 * rows + card * _bitmap_bytes(rows, 1.0 / card) + ids, "flops": 0}
        return {"bytes": ids + nq * card / 4.0 * _bitmap_bytes(rows, 1.0 / card), "flops": 0}
    if kind == "range":
        # both edge bins' bitmaps and values per query, and the index's
        # bitmaps once for all of them
        rows, bins, nq = case["rows"], case["bins"], case["queries"]
        edge = 2.0 * (_bitmap_bytes(rows, 1.0 / bins) + 4.0 * rows / bins)
        return {"bytes": nq * (8.0 + edge) + min(bins, nq * bins / 4.0) * _bitmap_bytes(rows, 1.0 / bins), "flops": 0}
    # conjunctions: each column's bitmaps once, each query's ids and count
    rows, nq, cap = case["rows"], case["queries"], case["cap"]
    cols = 2 * 1000 * _bitmap_bytes(rows, 1e-3) + 2 * 512 * _bitmap_bytes(rows, 1.0 / 512) + 8.0 * rows
    return {"bytes": min(1.0, nq / 8.0) * cols + nq * (8.0 + 4.0 * cap), "flops": 0}


def exact(case, seed):
    """Whole numbers only: nothing here has a value in 64 bits."""
    return None
