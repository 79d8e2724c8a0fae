"""The shared-memory kernel of plans without a compiled shape (wg_lowcard.cuh) against the
HBM-table path (WG_AGG_SMEM=0) over the forms it accepts: scalar, one-word, packed and
nullable keys, every aggregate kind it takes, projections, filters, selection vectors, join
types and index flavours, hints far below the groups, and sizes around a warp's and a CTA's step.

Integer and DECIMAL state must be equal; float sums are over non-negative values, so the
two summation orders differ by at most n * 2^-53 of the sum (below 1e-11 for these sizes)."""
import numpy as np
import pytest

from tests.helpers import assert_groups_equal

pytestmark = pytest.mark.gpu

I32, I64, F32, F64, DEC = 1, 2, 3, 4, 17
EMPTY = -0x7FFFFFFFFFFFFFFF
KINDS = ["sum_i", "sum_d", "sum_f", "avg_f", "min_f", "max_i", "count", "sum_f"]


def _columns(wg, n, seed, nulls):
    rng = np.random.default_rng(seed)
    ok = lambda p: rng.random(n) >= p if nulls else None  # noqa: E731
    k64 = rng.integers(0, 40, n).astype(np.int64) * 1_000_003
    k64[rng.random(n) < 0.05] = EMPTY
    k32 = rng.integers(-7, 8, n, dtype=np.int32)
    i64 = rng.integers(-(1 << 62), 1 << 62, n)
    dec = np.zeros(n, wg.DEC_DTYPE)
    lo = rng.integers(-(1 << 60), 1 << 60, n)
    dec["lo"] = lo.view(np.uint64)
    dec["hi"] = np.where(rng.random(n) < 0.3, rng.integers(-5, 5, n), lo >> 63)
    f32 = rng.random(n, dtype=np.float32)
    f32[rng.random(n) < 0.02] = np.inf
    f64 = rng.random(n)
    f64[rng.random(n) < 0.1] = 0.0
    small = rng.integers(0, 6, n, dtype=np.int32)
    return [wg.Column(I64, k64, ok(0.1)), wg.Column(I32, k32, ok(0.1)), wg.Column(I64, i64, ok(0.2)),
            wg.Column(DEC, dec, ok(0.2), scale=3), wg.Column(F32, f32, ok(0.2)), wg.Column(F64, f64, ok(0.2)),
            wg.Column(I32, small)]


def _both(ctx, monkeypatch, run):
    monkeypatch.setenv("WG_AGG_SMEM", "1")
    got = run()
    monkeypatch.setenv("WG_AGG_SMEM", "0")
    assert_groups_equal(got, run(), KINDS, rel=1e-11)


@pytest.mark.parametrize("nulls", [False, True])
@pytest.mark.parametrize("keys", [[], [0], [1], [6], [1, 6], [0, 6], [1, 6, 6]])
@pytest.mark.parametrize("n", [1, 33, 1025, 40_007])
def test_keys_and_sizes(ctx, monkeypatch, keys, nulls, n):
    import wadjet_b200 as wg
    cols = _columns(wg, n, n + len(keys), nulls)
    exprs = [wg.Expr(F64, [wg.Expr.col(5), wg.Expr.const_f(1.5), wg.Expr.col(6), "+", "*"]),
             wg.Expr(I64, [wg.Expr.col(2), wg.Expr.const_i(7), ">>", wg.Expr.const_i(255), "&"])]
    aggs = [wg.AggColumn(wg.AGG_SUM, 8), wg.AggColumn(wg.AGG_SUM, 3), wg.AggColumn(wg.AGG_SUM, 7),
            wg.AggColumn(wg.AGG_AVG, 5), wg.AggColumn(wg.AGG_MIN, 4), wg.AggColumn(wg.AGG_MAX, 2),
            wg.AggColumn(wg.AGG_COUNT, 4), wg.AggColumn(wg.AGG_SUM, 5)]
    rng = np.random.default_rng(n)
    sels = [None, np.flatnonzero(rng.random(n) < 0.6).astype(np.uint32)]
    for sel in sels:
        if sel is not None and len(sel) == 0:
            continue
        for hint in (1, 64, 700):  # 1: most keys find the CTA's table at its limit
            def run():
                a = wg.HashAggregate(ctx, keys, aggs, ndv_hint=hint)
                wg.run_pipeline(ctx, wg.Batch(cols, sel=sel), a, exprs=exprs,
                                filters=[(6, wg.OP_NE, 3), (5, wg.OP_LT, 0.95)])
                a.finalize()
                e = a.export()
                a.close()
                return e
            _both(ctx, monkeypatch, run)


@pytest.mark.parametrize("jtype", ["inner", "left", "semi", "anti"])
@pytest.mark.parametrize("key", ["dense", "direct", "hash32", "hash64"])
def test_joins(ctx, monkeypatch, jtype, key):
    import wadjet_b200 as wg
    n, b = 30_011, 700
    rng = np.random.default_rng(5)
    cols = _columns(wg, n, 9, True)
    ids = np.arange(b)
    if key.startswith("hash"):
        ids = ids % 300  # two or three build rows per key
    spread = {"dense": 1, "direct": 40_009, "hash32": 7, "hash64": 1 << 33}[key]
    typ, dt = (I64, np.int64) if key == "hash64" else (I32, np.int32)
    bkey = (ids * spread).astype(dt)
    group = (np.arange(b) % 23).astype(np.int32)
    fkey = (rng.integers(0, 2 * b if key != "hash64" else 600, n) * spread).astype(dt)
    pay = jtype in ("inner", "left")
    jt = {"inner": wg.abi.JOIN_INNER, "left": wg.abi.JOIN_LEFT, "semi": wg.abi.JOIN_SEMI, "anti": wg.abi.JOIN_ANTI}[jtype]
    join = wg.HashJoin(ctx, 0, 7, payload=[1] if pay else [], build_row_hint=b, join_type=jt)
    join.build([wg.Batch([wg.Column(typ, bkey), wg.Column(I32, group)])])
    cols.append(wg.Column(typ, fkey, rng.random(n) >= 0.05))
    gcol = 8 if pay else 6
    aggs = [wg.AggColumn(wg.AGG_SUM, 2), wg.AggColumn(wg.AGG_SUM, 3), wg.AggColumn(wg.AGG_SUM, 5),
            wg.AggColumn(wg.AGG_AVG, 5), wg.AggColumn(wg.AGG_MIN, 4), wg.AggColumn(wg.AGG_MAX, 2),
            wg.AggColumn(wg.AGG_COUNT, 4), wg.AggColumn(wg.AGG_SUM, 5)]
    for hint in (2, 40):
        def run():
            a = wg.HashAggregate(ctx, [gcol], aggs, ndv_hint=hint)
            wg.run_pipeline(ctx, wg.Batch(cols), a, join=join, filters=[(6, wg.OP_GE, 1)])
            a.finalize()
            e = a.export()
            a.close()
            return e
        _both(ctx, monkeypatch, run)
    join.close()


@pytest.mark.parametrize("nulls", [False, True])
@pytest.mark.parametrize("hint", [3700, 4000])
def test_one_cta_table_then_an_outgrown_hint(ctx, monkeypatch, nulls, hint):
    """Packed keys whose hint takes a whole SM's shared memory (5/8 to 3/4 of the slots), and
    far more groups than the memory table was sized for: the overflow's replays."""
    import wadjet_b200 as wg
    n = 1_000_003
    rng = np.random.default_rng(hint)
    ok = rng.random(n) >= 0.1 if nulls else None
    cols = [wg.Column(I32, rng.integers(0, 300, n, dtype=np.int32)), wg.Column(I32, rng.integers(0, 1000, n, dtype=np.int32)),
            wg.Column(I64, rng.integers(-(1 << 40), 1 << 40, n), ok)]

    def run():
        a = wg.HashAggregate(ctx, [0, 1], [wg.AggColumn(wg.AGG_SUM, 2), wg.AggColumn(wg.AGG_COUNT, 2)], ndv_hint=hint)
        wg.run_pipeline(ctx, wg.Batch(cols), a)
        a.finalize()
        e = a.export()
        a.close()
        return e

    monkeypatch.setenv("WG_AGG_SMEM", "1")
    got = run()
    monkeypatch.setenv("WG_AGG_SMEM", "0")
    assert_groups_equal(got, run(), ["sum_i", "count"])


def test_row_counters_of_a_skewed_join_key(ctx, monkeypatch):
    """One build key of 65,000 rows lets a CTA's share of the matches pass its 32-bit counters by
    the worst case, so a plan whose table takes a whole SM's shared memory leaves it."""
    import torch
    import wadjet_b200 as wg
    n, b, hot = 5_400_001, 4000, 65_000
    rng = np.random.default_rng(4)
    bkey = np.concatenate([np.arange(b), np.full(hot, b)]) * 977
    join = wg.HashJoin(ctx, 0, 0, payload=[1], build_row_hint=b + hot)
    join.build([wg.Batch([wg.Column(I64, bkey), wg.Column(I32, (np.arange(b + hot) % 7).astype(np.int32))])])
    fkey = torch.from_numpy(rng.integers(0, b, n) * 977).cuda()
    fkey[n // 2] = b * 977
    keys = [torch.from_numpy(rng.integers(0, m, n, dtype=np.int32)).cuda() for m in (50, 70)]
    val = torch.from_numpy(rng.integers(0, 1 << 40, n)).cuda()
    batch = wg.Batch([wg.Column(I64, fkey), wg.Column(I32, keys[0]), wg.Column(I32, keys[1]), wg.Column(I64, val)])

    def run():
        a = wg.HashAggregate(ctx, [1, 2], [wg.AggColumn(wg.AGG_SUM, 3), wg.AggColumn(wg.AGG_COUNT, -1)], ndv_hint=3700)
        wg.run_pipeline(ctx, batch, a, join=join, device=True)
        a.finalize()
        e = a.export()
        a.close()
        return e

    monkeypatch.setenv("WG_AGG_SMEM", "1")
    got = run()
    monkeypatch.setenv("WG_AGG_SMEM", "0")
    assert_groups_equal(got, run(), ["sum_i", "count"])
    join.close()


@pytest.mark.parametrize("jtype", [None, "left"])
@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("groups", [900, 30_000])
def test_groups_far_beyond_the_hint(ctx, monkeypatch, packed, groups, jtype):
    """Hints 10 to 10,000 times too low: rows without a slot, the second layout, the rows that
    find none there either, and chained join matches among them."""
    import wadjet_b200 as wg
    n = 300_007
    rng = np.random.default_rng(groups + packed)
    key = rng.integers(0, groups // (10 if packed else 1), n) * 1_000_003
    key[:50] = EMPTY
    cols = [wg.Column(I64, key, rng.random(n) >= 0.01), wg.Column(I32, rng.integers(0, 10, n, dtype=np.int32)),
            wg.Column(F64, rng.random(n), rng.random(n) >= 0.1), wg.Column(I64, rng.integers(-(1 << 40), 1 << 40, n)),
            wg.Column(I64, rng.integers(0, 600, n) * 7)]
    join, kw = None, {}
    if jtype:
        join = wg.HashJoin(ctx, 0, 4, payload=[1], build_row_hint=1200, join_type=wg.abi.JOIN_LEFT)
        join.build([wg.Batch([wg.Column(I64, np.arange(1000) % 400 * 7), wg.Column(I32, np.arange(1000, dtype=np.int32))])])
        kw["join"] = join
    aggs = [wg.AggColumn(wg.AGG_SUM, 2), wg.AggColumn(wg.AGG_SUM, 3), wg.AggColumn(wg.AGG_MAX, 3),
            wg.AggColumn(wg.AGG_COUNT, 5 if jtype else 2)]
    for hint in (3, 90, 900):
        def run():
            a = wg.HashAggregate(ctx, [0, 1] if packed else [0], aggs, ndv_hint=hint)
            wg.run_pipeline(ctx, wg.Batch(cols), a, filters=[(1, wg.OP_LT, 9)], **kw)
            a.finalize()
            e = a.export()
            a.close()
            return e
        monkeypatch.setenv("WG_AGG_SMEM", "1")
        got = run()
        monkeypatch.setenv("WG_AGG_SMEM", "0")
        assert_groups_equal(got, run(), ["sum_f", "sum_i", "max_i", "count"], rel=1e-11)
    if join:
        join.close()
