"""The queries that the engine is timed on, from one 2048-row batch to 2^28-row tables.

A case is one query (or one operator call) as a program that uses the package runs it: the
tables are on the GPU (Parquet pages on the host), the operators' handles exist, and a pass
resets the handles, runs the query and takes its finished rows. Sizes are those of the
workloads in ``bench.py`` and of their serving templates; rows come back in key order, as an
``ORDER BY`` would give them, because the device table lists its groups in no fixed order.

- ``listed()``   the cases by name;
- ``draw(rng)``  one more case of the same ranges;
- ``prepare``    tables and handles on the GPU, from the seed alone;
- ``run``        one pass;
- ``work``       the bytes one pass cannot do without;
- ``exact``      the same rows from plain torch and numpy.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import wadjet_b200 as wg
from wadjet_b200 import autotune, pages

I32, I64, F32, F64, DEC = wg.TYPE_INT32, wg.TYPE_INT64, wg.TYPE_FLOAT32, wg.TYPE_FLOAT64, wg.TYPE_DECIMAL
SUM, COUNT, MIN, MAX, AVG = wg.AGG_SUM, wg.AGG_COUNT, wg.AGG_MIN, wg.AGG_MAX, wg.AGG_AVG
CHUNK = 1 << 25          # rows generated at a time (bounds the generators' temporaries)
FIB = 0x9E3779B97F4A7C15  # odd: multiplying by it permutes the 64-bit integers


# ---------------------------------------------------------------------- cases --
def listed():
    return [
        # one record batch of the operator contract (2048 rows) through KernelFilter behind an
        # earlier filter's selection vector: what an operator-at-a-time host calls most often
        dict(name="filter_batch", kind="filter", rows=2048, type="int32", keep=0.8, nulls=0.0, selected=True),
        # KernelFilter over a whole resident int32 column, 80% of the rows kept
        dict(name="filter_scan", kind="filter", rows=1 << 28, type="int32", keep=0.8, nulls=0.0, selected=False),
        # the small dashboard query: GROUP BY over 2^20 rows, 4096 groups
        dict(name="groupby_small", kind="groupby", rows=1 << 20, groups=4096),
        # the same query over a 2^28-row table
        dict(name="groupby_large", kind="groupby", rows=1 << 28, groups=4096),
        # a pricing report over optional (nullable) columns: two small composite keys, seven
        # aggregates of mixed types, a projection; an odd row count
        dict(name="report_nullable", kind="report", rows=30_000_001, flags=3, states=2, nulls=0.05),
        # star join + aggregate, 2^28 facts x 2^22 dimension rows, join build included
        dict(name="starjoin_large", kind="starjoin", rows=1 << 28, dim=1 << 22, groups=1000),
        # LEFT join on sparse int64 keys with duplicate build rows and facts without a match
        dict(name="join_left", kind="join", rows=(1 << 24) + 3, build=1 << 20, dup=2, match=0.75, join="left"),
        # about as many groups as rows / 4 over a composite key, the groups handed over by owner
        # rank as the multi-GPU exchange does (DECIMAL sum, count, float MIN / MAX)
        dict(name="highcard_exchange", kind="highcard", rows=1 << 26, ids=1 << 24, parts=4),
        # network traffic by IPv4 /24 prefix: 65536 groups, the largest serving table
        dict(name="ipv4_prefix", kind="prefix", rows=100_000_000, hosts=24),
        # GROUP BY a URL-like string column, with the ten most frequent strings read back
        dict(name="string_keys", kind="strings", rows=20_000_003, distinct=100_000),
        # 64 small independent queries in one batched launch, every query's groups read back
        dict(name="batched", kind="batched", queries=64, min_rows=10_000, max_rows=10_000_000, max_card=4096),
        # a scan: dictionary and PLAIN Parquet pages with NULLs decoded from host memory, then
        # filtered and grouped
        dict(name="parquet_scan", kind="parquet", rows=(1 << 21) + 77, nulls=0.03),
    ]


def draw(rng):
    """One more case of the listed ranges (log-uniform sizes, odd ones among them)."""
    def size(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return min(hi, n | 1) if rng.random() < 0.5 else n

    kind = rng.choice(["filter", "groupby", "report", "starjoin", "join", "highcard", "prefix", "strings", "batched",
                       "parquet"])
    if kind == "filter":
        return dict(kind=kind, rows=size(2048, 1 << 28), type=rng.choice(["int32", "int64", "float32", "float64"]),
                    keep=round(rng.uniform(0.02, 0.98), 3), nulls=rng.choice([0.0, 0.0, 0.1]),
                    selected=rng.random() < 0.3)
    if kind == "groupby":
        return dict(kind=kind, rows=size(1 << 16, 1 << 28), groups=size(16, 1 << 15))
    if kind == "report":
        return dict(kind=kind, rows=size(1 << 16, 30_000_001), flags=rng.randint(2, 40), states=rng.randint(2, 50),
                    nulls=rng.choice([0.0, 0.01, 0.2]))
    if kind == "starjoin":
        return dict(kind=kind, rows=size(1 << 16, 1 << 28), dim=size(1 << 10, 1 << 22), groups=size(10, 2000))
    if kind == "join":
        return dict(kind=kind, rows=size(1 << 16, 1 << 24), build=size(1 << 10, 1 << 20), dup=rng.randint(1, 3),
                    match=round(rng.uniform(0.3, 1.0), 3), join=rng.choice(["inner", "left", "semi", "anti"]))
    if kind == "highcard":
        rows = size(1 << 22, 1 << 26)
        return dict(kind=kind, rows=rows, ids=max(1 << 20, rows // rng.randint(4, 8)), parts=rng.randint(4, 8))
    if kind == "prefix":
        return dict(kind=kind, rows=size(100_000, 100_000_000), hosts=rng.randint(20, 24))
    if kind == "strings":
        rows = size(1 << 18, 20_000_003)
        return dict(kind=kind, rows=rows, distinct=min(rows // 8, size(500, 100_000)))
    if kind == "batched":
        return dict(kind=kind, queries=rng.randint(16, 64), min_rows=10_000, max_rows=size(200_000, 10_000_000),
                    max_card=size(256, 4096))
    return dict(kind=kind, rows=size(1 << 16, (1 << 21) + 77), nulls=rng.choice([0.0, 0.03, 0.3]))


# ------------------------------------------------------------------- helpers --
_CTX = None


def _context():
    """The process's one context: its stream, its staging area and its HBM ledger."""
    global _CTX
    if _CTX is None:
        torch.cuda.init()
        _CTX = wg.Context(0)
    return _CTX


class State:
    """What a program holds between passes; the handles are destroyed with it."""

    def __init__(self, case, **kw):
        self.case = case
        self.handles = kw.pop("handles", [])
        self.__dict__.update(kw)

    def __del__(self):
        for h in self.handles:
            h.close()


def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1_000_003 + salt)
    return g


def _ints(g, lo, hi, n, dtype):
    """n integers in [lo, hi)."""
    out = torch.empty(n, dtype=dtype, device="cuda")
    for r in range(0, n, CHUNK):
        out[r:r + CHUNK].random_(lo, hi, generator=g)
    return out


def _floats(g, n, scale=1.0):
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    for r in range(0, n, CHUNK):
        out[r:r + CHUNK].uniform_(0.0, 1.0, generator=g)
    return out.mul_(scale) if scale != 1.0 else out


def _decimal(cents):
    """A DECIMAL column's 16-byte values {hi, lo} from int64 amounts."""
    out = torch.empty((cents.numel(), 2), dtype=torch.int64, device="cuda")
    out[:, 1] = cents
    out[:, 0] = cents >> 63
    return out


def _valid(g, n, share):
    """(validity words or None, bool per row or None): `share` of the rows are NULL."""
    if share <= 0.0:
        return None, None
    ok = torch.ones((n + 63) // 64 * 64, dtype=torch.bool, device="cuda")
    ok[:n] = torch.rand(n, generator=g, device="cuda") >= share
    bits = ok.view(-1, 8).to(torch.uint8)
    weight = torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], dtype=torch.uint8, device="cuda")
    return (bits * weight).sum(1, dtype=torch.uint8).view(torch.int64), ok[:n]


def _zipf(g, n, keys, perm, s=1.1):
    """n int32 keys, the rank's frequency falling as rank^-s, ranks spread by `perm`."""
    cdf = torch.cumsum(torch.arange(1, keys + 1, dtype=torch.float64, device="cuda").pow_(-s), 0)
    cdf /= cdf[-1].clone()
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    for r in range(0, n, CHUNK):
        u = torch.rand(min(CHUNK, n - r), generator=g, device="cuda", dtype=torch.float64)
        out[r:r + CHUNK] = perm[torch.searchsorted(cdf, u).clamp_(max=keys - 1)]
    return out


def _by_key(cols, base, span):
    """The rows of a query with one NOT NULL key in [base, base + span), in key order: each column
    (after the key) as an array over the key range, 0 where the key has no group."""
    at = cols[0][0].astype(np.int64) - base
    out = {}
    for i, (v, ok) in enumerate(cols[1:]):
        dense = np.zeros(span, v.dtype)
        dense[at] = v
        out["c%d" % i] = dense
    here = np.zeros(span, bool)
    here[at] = True
    out["present"] = here
    return out


def _sorted(cols, n_keys):
    """A query's rows in key order, NULLs last: {column: values, column validity}."""
    keys = []
    for v, ok in cols[:n_keys]:
        keys = [v, ~ok] + keys
    order = np.lexsort(keys)
    out = {}
    for i, (v, ok) in enumerate(cols):
        out["c%d" % i] = np.where(ok, v, 0)[order]
        out["ok%d" % i] = ok[order]
    return out


def _dense(present, **cols):
    """exact()'s counterpart of _by_key."""
    out = {k: torch.where(present, v, torch.zeros_like(v)) for k, v in cols.items()}
    out["present"] = present
    return out


def _sum_by(idx, val, n):
    """Sum of val per index in 64 bits (int64 or float64)."""
    out = torch.zeros(n, dtype=val.dtype, device=val.device)
    for r in range(0, idx.numel(), CHUNK):
        out.index_add_(0, idx[r:r + CHUNK].long(), val[r:r + CHUNK])
    return out


def _best_by(idx, val, n, how):
    lim = {"amin": torch.finfo(val.dtype).max if val.is_floating_point() else torch.iinfo(val.dtype).max,
           "amax": -torch.finfo(val.dtype).max if val.is_floating_point() else torch.iinfo(val.dtype).min}[how]
    out = torch.full((n,), lim, dtype=val.dtype, device=val.device)
    for r in range(0, idx.numel(), CHUNK):
        out.scatter_reduce_(0, idx[r:r + CHUNK].long(), val[r:r + CHUNK], how)
    return out


def _groups_arrays(n_keys, n_aggs, n, fields):
    """Host arrays for a raw export of the given fields, and the descriptor that names them."""
    kinds = {"keys": (n_keys, np.int64), "count": (n_aggs, np.int64), "i64": (n_aggs, np.int64),
             "f64": (n_aggs, np.float64)}
    a = {f: np.empty((kinds[f][0], n), kinds[f][1]) for f in fields}
    order = ("keys", "key_valid", "count", "i64", "f64", "dec", "has")
    return a, wg.abi.wg_group_export(*[a[f].ctypes.data if f in a else None for f in order])


# -------------------------------------------------------------------- filter --
_TORCH = {"int32": torch.int32, "int64": torch.int64, "float32": torch.float32, "float64": torch.float64}
_WG = {"int32": I32, "int64": I64, "float32": F32, "float64": F64}


def _filter_inputs(c, seed):
    g, n = _gen(seed), c["rows"]
    if c["type"].startswith("int"):
        col, value = _ints(g, 0, 1000, n, _TORCH[c["type"]]), int(1000 - round(1000 * c["keep"]))
    else:
        col = torch.rand(n, generator=g, device="cuda", dtype=_TORCH[c["type"]])
        value = float(1.0 - c["keep"])
    words, ok = _valid(g, n, c["nulls"])
    sel = None
    if c["selected"]:
        pick = torch.rand((n + 1) // 2, generator=g, device="cuda") < 0.5  # one row of each two
        sel = (torch.arange((n + 1) // 2, device="cuda") * 2 + pick).clamp_(max=n - 1).to(torch.int32)
    return col, value, words, ok, sel


def _filter_prepare(c, seed):
    ctx = _context()
    col, value, words, _, sel = _filter_inputs(c, seed)
    f = wg.KernelFilter(ctx, 0, wg.OP_GE, value)
    batch = wg.Batch([wg.Column(_WG[c["type"]], col, words)], sel=sel)
    out = torch.zeros(c["rows"] if sel is None else sel.numel(), dtype=torch.int32, device="cuda")
    return State(c, f=f, batch=batch, out=out, handles=[f])


def _filter_run(s):
    n = s.f.execute_device(s.batch, s.out)  # the selection is out[:n]; the rest stays zero
    return {"n": n, "sel": s.out}


def _filter_work(c):
    es = 8 if c["type"].endswith("64") else 4
    items = c["rows"] * (0.5 if c["selected"] else 1.0)
    return items * (es + (4 if c["selected"] else 0) + (0.125 if c["nulls"] else 0)) + \
        items * c["keep"] * (1 - c["nulls"]) * 4


def _filter_exact(c, seed):
    col, value, _, ok, sel = _filter_inputs(c, seed)
    keep = col >= value
    if ok is not None:
        keep &= ok
    rows = torch.nonzero(keep).view(-1).to(torch.int32) if sel is None else sel[keep[sel.long()]]
    out = torch.zeros(keep.numel() if sel is None else sel.numel(), dtype=torch.int32, device="cuda")
    out[:rows.numel()] = rows
    return {"n": rows.numel(), "sel": out}


# ------------------------------------------------------------------- groupby --
def _groupby_inputs(c, seed):
    g, n = _gen(seed), c["rows"]
    return (_ints(g, 0, c["groups"], n, torch.int64), _ints(g, 0, 1_000_000, n, torch.int64), _floats(g, n),
            _ints(g, 0, 10, n, torch.int32))


def _groupby_prepare(c, seed):
    k, v, f, flag = _groupby_inputs(c, seed)
    agg = wg.HashAggregate(_context(), [0], [wg.AggColumn(SUM, 1), wg.AggColumn(COUNT, -1), wg.AggColumn(MIN, 2),
                                             wg.AggColumn(MAX, 2)], ndv_hint=c["groups"])
    batch = wg.Batch([wg.Column(I64, k), wg.Column(I64, v), wg.Column(F64, f), wg.Column(I32, flag)])
    return State(c, agg=agg, batch=batch, handles=[agg])


def _groupby_run(s):
    s.agg.reset()
    wg.run_pipeline(_context(), s.batch, s.agg, filters=[(3, wg.OP_LT, 7)], device=True)
    s.agg.finalize()
    return _by_key(s.agg.collect(), 0, s.case["groups"])


def _groupby_work(c):
    return c["rows"] * 28 + c["groups"] * 40


def _groupby_exact(c, seed):
    k, v, f, flag = _groupby_inputs(c, seed)
    n = c["groups"]
    idx = torch.where(flag < 7, k, torch.full_like(k, n))  # dropped rows go to a group of their own
    cnt = _sum_by(idx, torch.ones_like(v), n + 1)[:n]
    return _dense(cnt > 0, c0=_sum_by(idx, v, n + 1)[:n].double(), c1=cnt,
                  c2=_best_by(idx, f, n + 1, "amin")[:n], c3=_best_by(idx, f, n + 1, "amax")[:n])


# -------------------------------------------------------------------- report --
def _report_inputs(c, seed):
    g, n = _gen(seed), c["rows"]
    flag, state = _ints(g, 0, c["flags"], n, torch.int32), _ints(g, 0, c["states"], n, torch.int32)
    qty, cents = _ints(g, 1, 51, n, torch.int64), _ints(g, 100, 10_000_001, n, torch.int64)
    disc, day = _floats(g, n, 0.1), _ints(g, 8000, 10_557, n, torch.int32)
    return flag, state, qty, cents, disc, day, _valid(g, n, c["nulls"]), _valid(g, n, c["nulls"])


def _report_prepare(c, seed):
    flag, state, qty, cents, disc, day, (pw, _), (dw, _) = _report_inputs(c, seed)
    expr = wg.Expr(F64, [wg.Expr.col(3), wg.Expr.const_f(1.0), wg.Expr.col(4), "-", "*"])
    agg = wg.HashAggregate(_context(), [0, 1],
                           [wg.AggColumn(SUM, 2), wg.AggColumn(SUM, 3), wg.AggColumn(SUM, 6), wg.AggColumn(AVG, 2),
                            wg.AggColumn(AVG, 4), wg.AggColumn(MAX, 5), wg.AggColumn(COUNT, -1)],
                           ndv_hint=c["flags"] * c["states"])
    batch = wg.Batch([wg.Column(I32, flag), wg.Column(I32, state), wg.Column(I64, qty),
                      wg.Column(DEC, _decimal(cents), pw, scale=2), wg.Column(F64, disc, dw),
                      wg.Column(wg.TYPE_DATE, day)])
    return State(c, agg=agg, batch=batch, expr=expr, handles=[agg])


def _report_run(s):
    s.agg.reset()
    wg.run_pipeline(_context(), s.batch, s.agg, filters=[(5, wg.OP_LE, 10_400)], exprs=[s.expr], device=True)
    s.agg.finalize()
    return _sorted(s.agg.collect(), 2)


def _report_work(c):
    return c["rows"] * (4 + 4 + 8 + 16 + 8 + 4 + (0.25 if c["nulls"] else 0.0)) + c["flags"] * c["states"] * 96


def _report_exact(c, seed):
    flag, state, qty, cents, disc, day, (_, pok), (_, dok) = _report_inputs(c, seed)
    m = c["flags"] * c["states"]
    idx = torch.where(day <= 10_400, flag.long() * c["states"] + state.long(), torch.full_like(qty, m))
    ok = torch.ones_like(day, dtype=torch.bool)
    pok, dok = (ok if pok is None else pok), (ok if dok is None else dok)
    zero = torch.zeros_like(disc)
    cnt = _sum_by(idx, ok.long(), m + 1)[:m]
    pcnt = _sum_by(idx, pok.long(), m + 1)[:m]
    dcnt = _sum_by(idx, dok.long(), m + 1)[:m]
    xcnt = _sum_by(idx, (pok & dok).long(), m + 1)[:m]
    price = cents.double() / 100.0
    cols = [(_sum_by(idx, qty, m + 1)[:m].double(), cnt),
            (_sum_by(idx, torch.where(pok, cents, torch.zeros_like(cents)), m + 1)[:m].double() / 100.0, pcnt),
            (_sum_by(idx, torch.where(pok & dok, price * (1.0 - disc), zero), m + 1)[:m], xcnt),
            (_sum_by(idx, qty, m + 1)[:m].double() / cnt.clamp(min=1), cnt),
            (_sum_by(idx, torch.where(dok, disc, zero), m + 1)[:m] / dcnt.clamp(min=1), dcnt),
            (_best_by(idx, day.long(), m + 1, "amax")[:m], cnt), (cnt, cnt)]
    at = torch.nonzero(cnt > 0).view(-1)
    out = {"c0": (at // c["states"]).to(torch.int32), "c1": (at % c["states"]).to(torch.int32),
           "ok0": torch.ones_like(at, dtype=torch.bool), "ok1": torch.ones_like(at, dtype=torch.bool)}
    for i, (v, n) in enumerate(cols):
        has = n[at] > 0
        out["c%d" % (i + 2)] = torch.where(has, v[at], torch.zeros_like(v[at]))
        out["ok%d" % (i + 2)] = has
    return out


# ------------------------------------------------------------------ starjoin --
def _starjoin_inputs(c, seed):
    g, n, d = _gen(seed), c["rows"], c["dim"]
    perm = torch.randperm(d, generator=g, device="cuda").to(torch.int32)
    key, grp = torch.randperm(d, generator=g, device="cuda").to(torch.int32), _ints(g, 0, c["groups"], d, torch.int32)
    return (_zipf(g, n, d, perm), _ints(g, 1, 51, n, torch.int32), _ints(g, 100, 10_000_001, n, torch.int64),
            _floats(g, n, 0.1), key, grp)


def _starjoin_prepare(c, seed):
    ctx = _context()
    fk, qty, cents, disc, key, grp = _starjoin_inputs(c, seed)
    join = wg.HashJoin(ctx, 0, 0, payload=[1], build_row_hint=c["dim"])
    agg = wg.HashAggregate(ctx, [4], [wg.AggColumn(SUM, 5), wg.AggColumn(SUM, 2)], ndv_hint=c["groups"])
    expr = wg.Expr(F64, [wg.Expr.col(2), wg.Expr.const_f(1.0), wg.Expr.col(3), "-", "*"])
    fact = wg.Batch([wg.Column(I32, fk), wg.Column(I32, qty), wg.Column(DEC, _decimal(cents), scale=2),
                     wg.Column(F64, disc)])
    dim = wg.Batch([wg.Column(I32, key), wg.Column(I32, grp)])
    return State(c, join=join, agg=agg, expr=expr, fact=fact, dim=dim, handles=[agg, join])


def _starjoin_run(s):
    s.join.reset()
    s.join.build([s.dim], device=True)
    s.agg.reset()
    wg.run_pipeline(_context(), s.fact, s.agg, filters=[(1, wg.OP_GT, 10)], join=s.join, exprs=[s.expr], device=True)
    s.agg.finalize()
    return _by_key(s.agg.collect(), 0, s.case["groups"])


def _starjoin_work(c):
    return c["rows"] * 32 + c["dim"] * 8 + c["groups"] * 40


def _starjoin_exact(c, seed):
    fk, qty, cents, disc, key, grp = _starjoin_inputs(c, seed)
    m = c["groups"]
    of = torch.empty_like(grp)
    of[key.long()] = grp
    cnt = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    dec, flt = torch.zeros_like(cnt), torch.zeros(m + 1, dtype=torch.float64, device="cuda")
    for r in range(0, c["rows"], CHUNK):
        w = slice(r, r + CHUNK)
        idx = torch.where(qty[w] > 10, of[fk[w].long()].long(), m)
        cnt += torch.bincount(idx, minlength=m + 1)
        dec += _sum_by(idx, cents[w], m + 1)
        flt += _sum_by(idx, (cents[w].double() / 100.0) * (1.0 - disc[w]), m + 1)
    return _dense(cnt[:m] > 0, c0=flt[:m], c1=dec[:m].double() / 100.0)


# ---------------------------------------------------------------------- join --
_JOINS = {"inner": wg.abi.JOIN_INNER, "left": wg.abi.JOIN_LEFT, "semi": wg.abi.JOIN_SEMI, "anti": wg.abi.JOIN_ANTI}
REGIONS = 50


def _spread(ids):
    """Sparse 63-bit keys of small ids."""
    return (ids * ctypes.c_int64(FIB).value) & 0x7FFFFFFFFFFFFFFF


def _join_inputs(c, seed):
    g, n, b = _gen(seed), c["rows"], c["build"]
    ids = max(1, b // c["dup"])
    bid = torch.arange(b, device="cuda", dtype=torch.int64) % ids
    region = _ints(g, 0, REGIONS, b, torch.int32)
    fid = _ints(g, 0, max(1, int(ids / c["match"])), n, torch.int64)
    return ids, bid, region, fid, _ints(g, 1, 51, n, torch.int32), _ints(g, 0, REGIONS, n, torch.int32), \
        _ints(g, 100, 10_000_001, n, torch.int64)


def _join_prepare(c, seed):
    ctx = _context()
    _, bid, region, fid, qty, grp, cents = _join_inputs(c, seed)
    pay = c["join"] in ("inner", "left")
    join = wg.HashJoin(ctx, 0, 0, payload=[1] if pay else [], build_row_hint=c["build"], join_type=_JOINS[c["join"]])
    agg = wg.HashAggregate(ctx, [4 if pay else 2], [wg.AggColumn(COUNT, -1), wg.AggColumn(SUM, 1), wg.AggColumn(SUM, 3),
                                                    wg.AggColumn(MAX, 3)], ndv_hint=REGIONS)
    fact = wg.Batch([wg.Column(I64, _spread(fid)), wg.Column(I32, qty), wg.Column(I32, grp), wg.Column(I64, cents)])
    build = wg.Batch([wg.Column(I64, _spread(bid)), wg.Column(I32, region)])
    return State(c, join=join, agg=agg, fact=fact, build=build, handles=[agg, join])


def _join_run(s):
    s.join.reset()
    s.join.build([s.build], device=True)
    s.agg.reset()
    wg.run_pipeline(_context(), s.fact, s.agg, filters=[(1, wg.OP_GT, 5)], join=s.join, device=True)
    s.agg.finalize()
    return _sorted(s.agg.collect(), 1)


def _join_work(c):
    pay = c["join"] in ("inner", "left")
    return c["rows"] * (20 if pay else 24) + c["build"] * (12 if pay else 8) + (REGIONS + 1) * 40


def _join_exact(c, seed):
    ids, bid, region, fid, qty, grp, cents = _join_inputs(c, seed)
    keep, hit, m = qty > 5, fid < ids, REGIONS + 1  # group REGIONS: the NULL key
    pairs = []
    if c["join"] in ("inner", "left"):
        of = torch.full((c["dup"] + 1, ids), -1, dtype=torch.int64, device="cuda")
        for d in range(c["dup"] + 1):  # build row d * ids + id, where there is one
            have = min(ids, max(0, c["build"] - d * ids))
            of[d, :have] = region[d * ids:d * ids + have].long()
        for d in range(c["dup"] + 1):
            r = of[d][fid.clamp(max=ids - 1)]
            pairs.append((keep & hit & (r >= 0), r))
        if c["join"] == "left":
            pairs.append((keep & ~hit, torch.full_like(fid, REGIONS)))
    else:
        pairs.append((keep & (hit if c["join"] == "semi" else ~hit), grp.long()))
    cnt, q, s = (torch.zeros(m, dtype=torch.int64, device="cuda") for _ in range(3))
    top = torch.full((m,), -1, dtype=torch.int64, device="cuda")
    for mask, r in pairs:
        at = torch.nonzero(mask).view(-1)
        cnt += torch.bincount(r[at], minlength=m)
        q += _sum_by(r[at], qty[at].long(), m)
        s += _sum_by(r[at], cents[at], m)
        top = torch.maximum(top, _best_by(r[at], cents[at], m, "amax"))
    at = torch.nonzero(cnt > 0).view(-1)
    null = at == REGIONS
    one = torch.ones_like(null)
    return {"c0": torch.where(null, 0, at).to(torch.int32), "ok0": ~null, "c1": cnt[at], "ok1": one,
            "c2": q[at].double(), "ok2": one, "c3": s[at].double(), "ok3": one, "c4": top[at], "ok4": one}


# ------------------------------------------------------------------ highcard --
HC_MUL = ctypes.c_int64(0xBF58476D1CE4E5B9).value          # b = id * HC_MUL (odd), so
HC_INV = ctypes.c_int64(pow(0xBF58476D1CE4E5B9, -1, 1 << 64)).value  # id = b * HC_INV


def _highcard_inputs(c, seed):
    g, n = _gen(seed), c["rows"]
    ids = _ints(g, 0, c["ids"], n, torch.int64)
    x = torch.empty(n, dtype=torch.float64, device="cuda")
    for r in range(0, n, CHUNK):
        x[r:r + CHUNK].normal_(generator=g)
    return ids, _ints(g, -100_000_000, 100_000_001, n, torch.int64), x


def _highcard_prepare(c, seed):
    ids, cents, x = _highcard_inputs(c, seed)
    agg = wg.HashAggregate(_context(), [0, 1], [wg.AggColumn(SUM, 2), wg.AggColumn(COUNT, -1), wg.AggColumn(MIN, 3),
                                                wg.AggColumn(MAX, 3)], ndv_hint=c["ids"])
    batch = wg.Batch([wg.Column(I32, (ids & 0xFFFF).to(torch.int32)), wg.Column(I64, ids * HC_MUL),
                      wg.Column(DEC, _decimal(cents), scale=2), wg.Column(F64, x)])
    return State(c, agg=agg, batch=batch, handles=[agg])


def _highcard_run(s):
    ctx = _context()
    with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream)):
        s.agg.reset()
        s.agg.consume(s.batch, device=True)
        rows, counts = s.agg.partition_state(s.case["parts"])
        # state rows by the key's id, a row of zeros where an id has no group
        table = torch.zeros((s.case["ids"], rows.shape[1]), dtype=torch.int64, device="cuda")
        table[rows[:, 1] * HC_INV] = rows
    return {"state": table, "part_rows": np.array(counts, np.int64)}


def _highcard_work(c):
    groups = c["ids"] * -math.expm1(-c["rows"] / c["ids"])
    return c["rows"] * 36 + groups * 72


def _ordered(v):
    """The order-preserving map of float64 onto 64-bit words that the state rows hold."""
    w = v.view(torch.int64)
    return torch.where(w < 0, ~w, w ^ torch.iinfo(torch.int64).min)


def _highcard_exact(c, seed):
    ids, cents, x = _highcard_inputs(c, seed)
    n = c["ids"]
    cnt = _sum_by(ids, torch.ones_like(ids), n)
    total = _sum_by(ids, cents, n)
    at = torch.arange(n, device="cuda", dtype=torch.int64)
    cols = [torch.zeros_like(at), at * HC_MUL, at & 0xFFFF, cnt, total, total >> 63,
            _ordered(_best_by(ids, x, n, "amin")), _ordered(_best_by(ids, x, n, "amax")), torch.zeros_like(at)]
    out = torch.stack(cols, 1)
    out[cnt == 0] = 0
    return {"state": out, "part_rows": None}


# -------------------------------------------------------------------- prefix --
ADDR0 = 10 << 24


def _prefix_inputs(c, seed):
    g, n = _gen(seed), c["rows"]
    addr = _ints(g, 0, 1 << c["hosts"], n, torch.int64).add_(ADDR0)
    nbytes = torch.empty(n, dtype=torch.int64, device="cuda")
    for r in range(0, n, CHUNK):
        m = min(CHUNK, n - r)
        z = torch.empty(m, dtype=torch.float64, device="cuda").normal_(8.0, 2.0, generator=g)
        nbytes[r:r + m] = z.exp_().round_().to(torch.int64)
    return addr, nbytes


def _prefix_prepare(c, seed):
    addr, nbytes = _prefix_inputs(c, seed)
    agg = wg.HashAggregate(_context(), [2], [wg.AggColumn(SUM, 1), wg.AggColumn(COUNT, -1)],
                           ndv_hint=1 << (c["hosts"] - 8))
    expr = wg.Expr(I64, [wg.Expr.col(0), wg.Expr.const_i(8), ">>"])
    batch = wg.Batch([wg.Column(wg.TYPE_IPV4, addr), wg.Column(I64, nbytes)])
    return State(c, agg=agg, batch=batch, expr=expr, handles=[agg])


def _prefix_run(s):
    s.agg.reset()
    wg.run_pipeline(_context(), s.batch, s.agg, exprs=[s.expr], device=True)
    s.agg.finalize()
    return _by_key(s.agg.collect(), ADDR0 >> 8, 1 << (s.case["hosts"] - 8))


def _prefix_work(c):
    return c["rows"] * 16 + (1 << (c["hosts"] - 8)) * 24


def _prefix_exact(c, seed):
    addr, nbytes = _prefix_inputs(c, seed)
    n = 1 << (c["hosts"] - 8)
    idx = (addr - ADDR0) >> 8
    cnt = _sum_by(idx, torch.ones_like(nbytes), n)
    return _dense(cnt > 0, c0=_sum_by(idx, nbytes, n).double(), c1=cnt)


# ------------------------------------------------------------------- strings --
TOP, LONGEST = 10, 56


def _most_frequent(count):
    """The ids of the TOP largest counts, the lower id first among equals."""
    n = len(count)
    rank = np.arange(n) - count * n
    top = np.argpartition(rank, TOP)[:TOP]
    return top[np.argsort(rank[top])]


def _padded(names):
    """Byte strings as rows of one array, zeros behind them."""
    return np.stack([np.frombuffer(b.ljust(LONGEST, b"\0"), np.uint8) for b in names])


def _string_inputs(c, seed):
    """(offsets, bytes, v, pick, the distinct strings' lengths, offsets and bytes): URL-like strings of
    8 to 56 bytes, the first five spelling the string's number, frequencies falling with the number."""
    g, n, d = _gen(seed), c["rows"], c["distinct"]
    lens = _ints(g, 8, 57, d, torch.int64)
    poff = torch.zeros(d + 1, dtype=torch.int64, device="cuda")
    poff[1:] = torch.cumsum(lens, 0)
    pool = _ints(g, 97, 123, int(poff[-1]), torch.uint8)
    ids = torch.arange(d, device="cuda", dtype=torch.int64)
    for k in range(5):
        pool[poff[:-1] + k] = (97 + (ids // (26 ** k)) % 26).to(torch.uint8)
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    pick = (u.square_() * d).to(torch.int64).clamp_(max=d - 1)
    offs = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    offs[1:] = torch.cumsum(lens[pick], 0)
    raw = torch.empty(int(offs[-1]), dtype=torch.uint8, device="cuda")
    step = 1 << 22
    for r in range(0, n, step):
        e = min(n, r + step)
        b0, b1 = int(offs[r]), int(offs[e])
        shift = torch.repeat_interleave(poff[pick[r:e]] - offs[r:e], lens[pick[r:e]])
        raw[b0:b1] = pool[shift.add_(torch.arange(b0, b1, device="cuda", dtype=torch.int64))]
    return offs.to(torch.int32), raw, _ints(g, 0, 1_000_000, n, torch.int64), pick, lens, poff, pool


def _strings_prepare(c, seed):
    offs, raw, v = _string_inputs(c, seed)[:3]
    agg = wg.HashAggregate(_context(), [0], [wg.AggColumn(COUNT, -1), wg.AggColumn(SUM, 1)])
    batch = wg.Batch([wg.Column(wg.TYPE_BYTES, (offs, raw)), wg.Column(I64, v)])
    return State(c, agg=agg, batch=batch, handles=[agg])


def _strings_run(s):
    s.agg.reset()
    s.agg.consume(s.batch, device=True)
    n = s.agg.finalize()
    a, e = _groups_arrays(1, 2, n, ("keys", "count", "i64"))
    wg._check(wg.lib.wg_agg_export(s.agg.h, ctypes.byref(e)))
    count, total = np.empty(n, np.int64), np.empty(n, np.int64)
    count[a["keys"][0]] = a["count"][0]  # ids number the strings by first appearance
    total[a["keys"][0]] = a["i64"][1]
    best = _most_frequent(count)
    names = s.agg.key_strings(best)
    return {"count": count, "sum": total, "top": best, "text": _padded(names)}


def _strings_work(c):
    return c["rows"] * (4 + 32 + 8) + c["distinct"] * (32 + 24)


def _strings_exact(c, seed):
    offs, raw, v, pick, lens, poff, pool = _string_inputs(c, seed)
    d = c["distinct"]
    row = torch.arange(c["rows"], device="cuda", dtype=torch.int64)
    first = _best_by(pick, row, d, "amin")
    order = torch.argsort(first)
    order = order[first[order] < c["rows"]]  # the strings that occur, by first appearance
    count, total = torch.bincount(pick, minlength=d)[order], _sum_by(pick, v, d)[order]
    best = _most_frequent(count.cpu().numpy())
    names = [pool[poff[i]:poff[i + 1]].cpu().numpy().tobytes() for i in order.cpu().numpy()[best]]
    return {"count": count, "sum": total, "top": best, "text": _padded(names)}


# ------------------------------------------------------------------- batched --
def _batched_shape(c):
    """(rows, key cardinality, filter threshold) of each query: sizes spread over their ranges."""
    q = c["queries"]
    for i in range(q):
        a, b = (i + 0.5) / q, ((i * 37) % q + 0.5) / q
        yield (int(c["min_rows"] * (c["max_rows"] / c["min_rows"]) ** a), int(16 * (c["max_card"] / 16) ** b),
               100 + (i * 53) % 801)


def _batched_inputs(c, seed, i, n, card):
    g = _gen(seed, i)
    val = _ints(g, 0, 1_000_000, n, torch.int64) if i % 2 == 0 else _floats(g, n)
    return _ints(g, 0, card, n, torch.int64), val, _ints(g, 0, 1000, n, torch.int32)


def _batched_prepare(c, seed):
    ctx, queries = _context(), []
    for i, (n, card, thr) in enumerate(_batched_shape(c)):
        key, val, filt = _batched_inputs(c, seed, i, n, card)
        queries.append(dict(batch=wg.Batch([wg.Column(I64, key), wg.Column(I64 if i % 2 == 0 else F64, val),
                                            wg.Column(I32, filt)]), group_by=[0], ndv_hint=card,
                            aggs=[wg.AggColumn(SUM, 1), wg.AggColumn(COUNT, -1), wg.AggColumn(MIN, 1),
                                  wg.AggColumn(MAX, 1)], filters=[(2, wg.OP_LT, thr)], keep=(key, val, filt)))
    torch.cuda.synchronize()
    b = wg.BatchedQueries(ctx, queries, params=autotune.load_tuned())
    cards = [card for _, card, _ in _batched_shape(c)]
    return State(c, b=b, queries=queries, base=np.concatenate([[0], np.cumsum(cards)]), handles=[b])


def _batched_run(s):
    groups = s.b.run()
    total = int(s.base[-1])
    count, ints, floats = np.zeros(total, np.int64), np.zeros((3, total), np.int64), np.zeros((3, total))
    for q, n in enumerate(groups):
        field, out = ("i64", ints) if q % 2 == 0 else ("f64", floats)
        a, e = _groups_arrays(1, 4, int(n), ("keys", "count", field))
        if n:
            wg._check(wg.lib.wg_batched_export(s.b.h, q, ctypes.byref(e)))
        at = a["keys"][0] + s.base[q]
        count[at] = a["count"][1]
        for k, col in enumerate((0, 2, 3)):
            out[k, at] = a[field][col]
    return {"groups": groups, "count": count, "ints": ints, "floats": floats}


def _batched_work(c):
    return sum(n * 20 + card * 40 for n, card, _ in _batched_shape(c))


def _batched_exact(c, seed):
    groups, counts, ints, floats = [], [], [], []
    for i, (n, card, thr) in enumerate(_batched_shape(c)):
        key, val, filt = _batched_inputs(c, seed, i, n, card)
        idx = torch.where(filt < thr, key, torch.full_like(key, card))
        cnt = _sum_by(idx, torch.ones_like(key), card + 1)[:card]
        cols = torch.stack([_sum_by(idx, val, card + 1)[:card], _best_by(idx, val, card + 1, "amin")[:card],
                            _best_by(idx, val, card + 1, "amax")[:card]])
        cols = torch.where(cnt > 0, cols, torch.zeros_like(cols))
        groups.append(int((cnt > 0).sum()))
        counts.append(cnt)
        ints.append(cols if i % 2 == 0 else torch.zeros_like(cols, dtype=torch.int64))
        floats.append(cols if i % 2 else torch.zeros_like(cols, dtype=torch.float64))
    return {"groups": np.array(groups, np.int64), "count": torch.cat(counts), "ints": torch.cat(ints, 1),
            "floats": torch.cat(floats, 1)}


# ------------------------------------------------------------------- parquet --
PAGE_ROWS = 1 << 17
STORES = 1000
RUN = 504  # values of one bit-packed run, as Parquet writers cut them


def _hybrid(v, bw):
    """Values below 2^bw as bit-packed runs of at most 504 values."""
    out = b""
    full = len(v) // RUN * RUN
    for part, groups in ((v[:full], RUN // 8), (v[full:], (len(v) - full + 7) // 8)):
        if not len(part):
            continue
        part = np.concatenate([part, np.zeros(-len(part) % 8, part.dtype)])
        bits = ((part[:, None] >> np.arange(bw)) & 1).astype(np.uint8)
        body = np.packbits(bits.reshape(-1), bitorder="little").reshape(-1, groups * bw)
        out += np.concatenate([np.full((len(body), 1), groups << 1 | 1, np.uint8), body], 1).tobytes()
    return out


def _parquet_inputs(c, seed):
    r, n = np.random.default_rng(seed), c["rows"]
    return (r.integers(0, STORES, n, dtype=np.int32), r.integers(0, 2557, n, dtype=np.int32),
            r.integers(-10_000_000, 10_000_001, n, dtype=np.int64), r.integers(0, 50, n, dtype=np.int32),
            r.random(n), r.random(n) >= c["nulls"], r.random(n) >= c["nulls"])


def _chunk(type_id, values, ok=None, dictionary=None, scale=0):
    ps = []
    bw = 0 if dictionary is None else max(1, (len(dictionary) - 1).bit_length())
    for r0 in range(0, len(values), PAGE_ROWS):
        v, levels = values[r0:r0 + PAGE_ROWS], None
        if ok is not None:
            levels = _hybrid(ok[r0:r0 + PAGE_ROWS].astype(np.uint8), 1)
            v = v[ok[r0:r0 + PAGE_ROWS]]
        data = v.tobytes() if dictionary is None else bytes([bw]) + _hybrid(v, bw)
        ps.append(pages.Page(min(PAGE_ROWS, len(values) - r0), data,
                             pages.ENC_PLAIN if dictionary is None else pages.ENC_RLE_DICTIONARY, levels))
    return pages.Chunk(type_id, ps, scale, dictionary)


def _parquet_prepare(c, seed):
    store, day, cents, qty, price, aok, qok = _parquet_inputs(c, seed)
    null = c["nulls"] > 0
    chunks = [_chunk(I32, store, dictionary=np.arange(STORES, dtype=np.int32)),
              _chunk(wg.TYPE_DATE, day, dictionary=np.arange(8000, 8000 + 2557, dtype=np.int32)),
              _chunk(DEC, cents, aok if null else None, scale=2),
              _chunk(I32, qty, qok if null else None, dictionary=np.arange(1, 51, dtype=np.int32)),
              _chunk(F64, price)]
    agg = wg.HashAggregate(_context(), [0], [wg.AggColumn(SUM, 2), wg.AggColumn(SUM, 3), wg.AggColumn(AVG, 4),
                                             wg.AggColumn(COUNT, -1)], ndv_hint=STORES)
    return State(c, chunks=chunks, agg=agg, handles=[agg])


def _parquet_run(s):
    ctx = _context()
    batch = wg.DeviceBatch.decode(ctx, s.chunks)
    try:
        s.agg.reset()
        wg.run_pipeline(ctx, batch, s.agg, filters=[(1, wg.OP_LT, 10_000)], device=True)
        s.agg.finalize()
        return _by_key(s.agg.collect(), 0, STORES)
    finally:
        batch.close()


def _parquet_work(c):
    return c["rows"] * ((10 + 12 + 6) / 8 + 8 + 8 + (0.25 if c["nulls"] else 0.0)) + STORES * 40


def _parquet_exact(c, seed):
    store, day, cents, qty, price, aok, qok = _parquet_inputs(c, seed)
    if c["nulls"] <= 0:
        aok, qok = np.ones_like(aok), np.ones_like(qok)
    keep = day + 8000 < 10_000
    store, cents, qty, price, aok, qok = (a[keep] for a in (store, cents, qty, price, aok, qok))
    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    idx = t(store)
    cnt = _sum_by(idx, torch.ones_like(idx, dtype=torch.int64), STORES)
    return _dense(cnt > 0, c0=_sum_by(idx, t(np.where(aok, cents, 0)), STORES).double() / 100.0,
                  c1=_sum_by(idx, t(np.where(qok, qty.astype(np.int64) + 1, 0)), STORES).double(),
                  c2=_sum_by(idx, t(price), STORES) / cnt.clamp(min=1), c3=cnt)


# -------------------------------------------------------------------- entry --
_KINDS = {k: tuple(globals()["_%s_%s" % (k, f)] for f in ("prepare", "run", "work", "exact"))
          for k in ("filter", "groupby", "report", "starjoin", "join", "highcard", "prefix", "strings", "batched",
                    "parquet")}


def prepare(case, seed):
    s = _KINDS[case["kind"]][0](case, seed)
    torch.cuda.synchronize()  # the tables are complete before another stream reads them
    return s


def run(state):
    return _KINDS[state.case["kind"]][1](state)


def work(case):
    return {"bytes": float(_KINDS[case["kind"]][2](case)), "flops": 0.0}


def exact(case, seed):
    return _KINDS[case["kind"]][3](case, seed)
