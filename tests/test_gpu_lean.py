"""The row loop of compiled one-key group-by shapes (wg_lean.cuh) against the HBM-table path
(WG_AGG_SMEM=0): keys of a small range (slot = key - base), sparse keys (hashed), a range with
rows outside the sampled window, the key equal to the empty pattern, more groups than the hint
gives room for, float SUM inputs of widely different magnitude (fixed point and its float
fallback), and sizes around a lane's, a warp's and a CTA's rows.

Integer state and MIN / MAX must be equal. Float sums: at most n additions of non-negative
values in any order, so two orders differ by at most n * 2^-53 of the sum (below 1e-10 here);
the infinite and NaN inputs must give the same infinities and NaNs."""
import numpy as np
import pytest

from tests.helpers import canonical_order

pytestmark = pytest.mark.gpu

I32, I64, F64 = 1, 2, 4
EMPTY = -0x7FFFFFFFFFFFFFFF


def _keys(kind, n, rng):
    if kind == "dense":
        return rng.integers(-3000, 1000, n)
    if kind == "sparse":
        return rng.integers(0, 3000, n) * 0x1234567891
    if kind == "outliers":  # nearly all keys in one range, a few far away on both sides
        k = rng.integers(500, 900, n)
        k[rng.random(n) < 0.002] = 1 << 62
        k[rng.random(n) < 0.002] = -(1 << 62)
        return k
    if kind == "empty":
        k = rng.integers(0, 50, n) + EMPTY - 10
        return k
    return rng.integers(0, 60_000, n)  # "many": more groups than the hint


def _values(kind, n, rng):
    if kind == "int":
        return rng.integers(-(1 << 62), 1 << 62, n)
    if kind == "wide":  # magnitudes over 2^-300 .. 2^300, zeros among them
        return np.where(rng.random(n) < 0.1, 0.0, np.ldexp(rng.random(n), rng.integers(-300, 300, n)))
    v = rng.random(n) * 1e5
    if kind == "special":
        v[rng.random(n) < 0.001] = np.inf
        v[rng.random(n) < 0.0005] = np.nan
    return v


def _run(ctx, wg, shape, cols, hint, n):
    key, val, filt = cols
    if shape == "groupby":  # flag, k, v, f
        a = wg.HashAggregate(ctx, [0], [wg.AggColumn(wg.AGG_SUM, 1), wg.AggColumn(wg.AGG_COUNT, -1),
                                        wg.AggColumn(wg.AGG_MIN, 3), wg.AggColumn(wg.AGG_MAX, 3)], ndv_hint=hint)
        batch = wg.Batch([wg.Column(I64, key), wg.Column(I64, np.arange(n)), wg.Column(I32, filt), wg.Column(F64, val)])
    else:
        a = wg.HashAggregate(ctx, [0], [wg.AggColumn(wg.AGG_SUM, 1), wg.AggColumn(wg.AGG_COUNT, -1),
                                        wg.AggColumn(wg.AGG_MIN, 1), wg.AggColumn(wg.AGG_MAX, 1)], ndv_hint=hint)
        batch = wg.Batch([wg.Column(I64, key), wg.Column(I64 if shape == "i64" else F64, val), wg.Column(I32, filt)])
    wg.run_pipeline(ctx, batch, a, filters=[(2, wg.OP_LT, 7)])
    a.finalize()
    assert a.kernel_shape == {"groupby": 2, "i64": 4, "f64": 5}[shape]
    e = a.export()
    a.close()
    return e


@pytest.mark.parametrize("shape,values", [("groupby", "float"), ("i64", "int"), ("f64", "float"), ("f64", "wide"),
                                          ("f64", "special")])
@pytest.mark.parametrize("keys", ["dense", "sparse", "outliers", "empty", "many"])
@pytest.mark.parametrize("n", [1, 127, 129, 4097, 100_003])
def test_lean_equals_the_hbm_table(ctx, monkeypatch, shape, values, keys, n):
    import wadjet_b200 as wg
    rng = np.random.default_rng(n + len(keys) * 7 + len(values))
    cols = (_keys(keys, n, rng).astype(np.int64), _values(values, n, rng), rng.integers(0, 10, n, dtype=np.int32))
    hint = 2000 if keys == "many" else 4000
    monkeypatch.setenv("WG_AGG_SMEM", "1")
    got = _run(ctx, wg, shape, cols, hint, n)
    monkeypatch.setenv("WG_AGG_SMEM", "0")
    want = _run(ctx, wg, shape, cols, hint, n)
    og, ow = canonical_order(got), canonical_order(want)
    for f in ("keys", "count", "i64", "has"):
        np.testing.assert_array_equal(got[f][:, og], want[f][:, ow])
    g, w = got["f64"][:, og], want["f64"][:, ow]
    np.testing.assert_array_equal(g[2:], w[2:])  # MIN, MAX
    if shape == "f64":
        np.testing.assert_array_equal(np.isnan(g[0]), np.isnan(w[0]))
        np.testing.assert_array_equal(np.isinf(g[0]), np.isinf(w[0]))
        fin = np.isfinite(w[0])
        assert (np.abs(g[0][fin] - w[0][fin]) <= 1e-10 * np.abs(w[0][fin])).all()


@pytest.mark.parametrize("limit", [1024, 4096])
def test_batched_lean_equals_the_hbm_table(ctx, limit):
    """The same row loop for the work items of a batch: queries in shared tables of two CTAs per
    SM or one, and queries in HBM beside them (a launch each), against a batch whose tables are
    all in HBM. A result is read twice (the second without a run in between)."""
    import torch
    import wadjet_b200 as wg
    rng = np.random.default_rng(limit)
    queries = []
    for i, (keys, n, hint) in enumerate([("dense", 100_003, 4000), ("sparse", 40_001, 3000), ("outliers", 4097, 900),
                                         ("empty", 129, 50), ("many", 150_001, 2000), ("sparse", 1, 16),
                                         ("many", 70_000, 30_000), ("dense", 66_000, 4000)]):
        val = _values("int", n, rng) if i % 2 == 0 else _values(["wide", "special", "float", "float"][i // 2], n, rng)
        cols = [torch.from_numpy(x).cuda() for x in
                (_keys(keys, n, rng).astype(np.int64), val, rng.integers(0, 10, n, dtype=np.int32))]
        queries.append(dict(batch=wg.Batch([wg.Column(I64, cols[0]), wg.Column(I64 if i % 2 == 0 else F64, cols[1]),
                                            wg.Column(I32, cols[2])]), group_by=[0], ndv_hint=hint,
                            aggs=[wg.AggColumn(wg.AGG_SUM, 1), wg.AggColumn(wg.AGG_COUNT, -1),
                                  wg.AggColumn(wg.AGG_MIN, 1), wg.AggColumn(wg.AGG_MAX, 1)],
                            filters=[(2, wg.OP_LT, 7)], keep=cols))
    torch.cuda.synchronize()
    out = []
    for params in (wg.TuneParams(tile_rows=32768, smem_max_groups=limit), wg.TuneParams(smem_max_groups=-1)):
        b = wg.BatchedQueries(ctx, queries, params)
        for _ in range(2):  # the first run may re-run queries with more groups than their hint
            counts = b.run()
        res = [b.export(q, int(c)) for q, c in enumerate(counts)]
        again = b.export(0, int(counts[0]))
        np.testing.assert_array_equal(np.sort(again["keys"][0]), np.sort(res[0]["keys"][0]))
        out.append(res)
        b.close()
    for i, (got, want) in enumerate(zip(*out)):
        og, ow = canonical_order(got), canonical_order(want)
        for f in ("keys", "count", "i64", "has"):
            np.testing.assert_array_equal(got[f][:, og], want[f][:, ow])
        g, w = got["f64"][:, og], want["f64"][:, ow]
        np.testing.assert_array_equal(g[2:], w[2:])
        np.testing.assert_array_equal(np.isnan(g[0]), np.isnan(w[0]))
        np.testing.assert_array_equal(np.isinf(g[0]), np.isinf(w[0]))
        fin = np.isfinite(w[0])
        assert (np.abs(g[0][fin] - w[0][fin]) <= 1e-10 * np.abs(w[0][fin])).all()


def _same_groups(got, want, floats):
    """Groups equal to the HBM-table path's, by the bounds of the module's first lines."""
    og, ow = canonical_order(got), canonical_order(want)
    for f in ("keys", "count", "i64", "has"):
        np.testing.assert_array_equal(got[f][:, og], want[f][:, ow])
    g, w = got["f64"][:, og], want["f64"][:, ow]
    np.testing.assert_array_equal(g[2:], w[2:])
    if floats:
        assert (np.abs(g[0] - w[0]) <= 1e-10 * np.abs(w[0])).all()


def _ten_thousand(spread, n, rng):
    return rng.integers(0, 10_000, n) * (1 if spread == "dense" else 0x1234567891)


@pytest.mark.parametrize("hint", [16, 100])
@pytest.mark.parametrize("keys", ["dense", "sparse"])
@pytest.mark.parametrize("shape", ["groupby", "i64", "f64"])
def test_hint_far_below_the_groups(ctx, monkeypatch, shape, keys, hint):
    """A hint two orders below 10,000 groups: every CTA meets more keys than its table takes, so
    the table reaches its limit and the probes of absent keys end there."""
    import wadjet_b200 as wg
    n = 400_003
    rng = np.random.default_rng(hint)
    cols = (_ten_thousand(keys, n, rng).astype(np.int64), _values("int" if shape == "i64" else "float", n, rng),
            rng.integers(0, 10, n, dtype=np.int32))
    monkeypatch.setenv("WG_AGG_SMEM", "1")
    got = _run(ctx, wg, shape, cols, hint, n)
    monkeypatch.setenv("WG_AGG_SMEM", "0")
    _same_groups(got, _run(ctx, wg, shape, cols, hint, n), shape == "f64")


@pytest.mark.parametrize("hint", [16, 100])
@pytest.mark.parametrize("keys", ["dense", "sparse"])
def test_batched_hint_far_below_the_groups(ctx, keys, hint):
    """The same for work items, whose tables have 256 slots for such hints: first runs (the rows
    of an item into its small table, then the query again alone) and the run after them."""
    import torch
    import wadjet_b200 as wg
    rng = np.random.default_rng(hint + 1)
    queries = []
    for i, n in enumerate([200_003, 90_001, 40_000]):
        val = _values("int" if i % 2 == 0 else "float", n, rng)
        cols = [torch.from_numpy(x).cuda() for x in
                (_ten_thousand(keys, n, rng).astype(np.int64), val, rng.integers(0, 10, n, dtype=np.int32))]
        queries.append(dict(batch=wg.Batch([wg.Column(I64, cols[0]), wg.Column(I64 if i % 2 == 0 else F64, cols[1]),
                                            wg.Column(I32, cols[2])]), group_by=[0], ndv_hint=hint,
                            aggs=[wg.AggColumn(wg.AGG_SUM, 1), wg.AggColumn(wg.AGG_COUNT, -1),
                                  wg.AggColumn(wg.AGG_MIN, 1), wg.AggColumn(wg.AGG_MAX, 1)],
                            filters=[(2, wg.OP_LT, 7)], keep=cols))
    torch.cuda.synchronize()
    out = []
    for params in (wg.TuneParams(tile_rows=32768), wg.TuneParams(smem_max_groups=-1)):
        b = wg.BatchedQueries(ctx, queries, params)
        res = []
        for _ in range(2):
            counts = b.run()
            res.append([b.export(q, int(c)) for q, c in enumerate(counts)])
        out.append(res)
        b.close()
    for got_run, want_run in zip(*out):
        for i, (got, want) in enumerate(zip(got_run, want_run)):
            _same_groups(got, want, i % 2 == 1)


def _magnitudes(n, groups, rng):
    """Keys and positive values, one power of two per group: 2^-1000, 2^-500, 1, 2^500 or 2^990."""
    key = rng.integers(0, groups, n)
    return key, np.ldexp(rng.random(n) + 0.5, np.array([-1000, -500, 0, 500, 990])[key % 5])


def _sums_close(e, key, val, keep):
    """Each group's SUM within the rounding of its rows' additions in any order."""
    order = np.argsort(e["keys"][0])
    want = np.zeros(key.max() + 1)
    np.add.at(want, key[keep], val[keep])
    np.testing.assert_array_equal(e["keys"][0][order], np.unique(key[keep]))
    want = want[np.unique(key[keep])]
    assert (np.abs(e["f64"][0][order] - want) <= 1e-10 * want).all()


@pytest.mark.parametrize("groups", [7, 300])
def test_groups_of_small_values_beside_huge_ones(ctx, monkeypatch, groups):
    """Groups whose values underflow at the scale that another group's values set: they add in
    binary64. Plain and batched; the scale may also come from a row that the filter drops."""
    import torch
    import wadjet_b200 as wg
    monkeypatch.setenv("WG_AGG_SMEM", "1")
    n = 50_003
    rng = np.random.default_rng(groups)
    key, val = _magnitudes(n, groups, rng)
    filt = rng.integers(0, 10, n, dtype=np.int32)
    filt[key % 5 == 4] = 9  # the huge values are dropped in the second query
    for f in (np.zeros(n, np.int32), filt):
        _sums_close(_run(ctx, wg, "f64", (key, val, f), 400, n), key, val, f < 7)
    cols = [torch.from_numpy(x).cuda() for x in (key, val, filt)]
    b = wg.BatchedQueries(ctx, [dict(batch=wg.Batch([wg.Column(I64, cols[0]), wg.Column(F64, cols[1]),
                                                     wg.Column(I32, cols[2])]), group_by=[0], ndv_hint=400,
                                     aggs=[wg.AggColumn(wg.AGG_SUM, 1), wg.AggColumn(wg.AGG_COUNT, -1),
                                           wg.AggColumn(wg.AGG_MIN, 1), wg.AggColumn(wg.AGG_MAX, 1)],
                                     filters=[(2, wg.OP_LT, lim)]) for lim in (10, 7)])
    counts = b.run()
    for q, lim in enumerate((10, 7)):
        _sums_close(b.export(q, int(counts[q])), key, val, filt < lim)
    b.close()


def test_star_join_small_products_beside_huge_ones(ctx):
    """The same in the star join's SUM(price * (1 - disc)): products near 2^-152 in every group
    but one, whose products near 2^1005 set the scale."""
    import torch
    import wadjet_b200 as wg
    rng = np.random.default_rng(6)
    nd, n = 1 << 12, 40_003
    grp = (np.arange(nd) % 50).astype(np.int32)
    fk = rng.integers(0, nd, n).astype(np.int32)
    huge = grp[fk] == 0
    price = np.zeros(n, wg.DEC_DTYPE)  # units of 10^-30: 2^126 or 1
    price["hi"], price["lo"] = np.where(huge, 1 << 62, 0), np.where(huge, 0, 1)
    disc = np.where(huge, -(2.0 ** 979), 1.0 - 2.0 ** -53)
    qty = np.full(n, 20, np.int32)
    j = wg.HashJoin(ctx, 0, 0, payload=[1], build_row_hint=nd)
    j.build([wg.Batch([wg.Column(I32, np.arange(nd, dtype=np.int32)), wg.Column(I32, grp)])])
    g = wg.HashAggregate(ctx, [4], [wg.AggColumn(wg.AGG_SUM, 5), wg.AggColumn(wg.AGG_SUM, 2)], ndv_hint=50)
    dev = [torch.from_numpy(x).cuda() for x in (fk, qty, price.view(np.int64).reshape(-1, 2), disc)]
    batch = wg.Batch([wg.Column(I32, dev[0]), wg.Column(I32, dev[1]), wg.Column(17, dev[2], scale=30),
                      wg.Column(F64, dev[3])])
    wg.run_pipeline(ctx, batch, g, filters=[(1, wg.OP_GT, 10)], join=j, device=True,
                    exprs=[wg.Expr(F64, [wg.Expr.col(2), wg.Expr.const_f(1.0), wg.Expr.col(3), "-", "*"])])
    g.finalize()
    assert g.kernel_shape == 1
    e = g.export()
    rows = np.bincount(grp[fk], minlength=50)
    one = np.where(np.arange(50) == 0, float(1 << 126) / 1e30 * (1.0 + 2.0 ** 979), 1.0 / 1e30 * 2.0 ** -53)
    want = (rows * one)[e["keys"][0]]
    assert (np.abs(e["f64"][0] - want) <= 1e-10 * want).all()
    g.close()
    j.close()
