"""Key windows (wg_window.cuh) against the hash-table path (WG_KEY_WINDOW=0): compiled and
interpreted plans, keys of a known and of a sampled range, rows outside the window, NULL keys,
ranges and key frequencies that take no window, a selection vector, DECIMAL MIN / MAX, and a
second batch into the same aggregate.

Integer and DECIMAL state and MIN / MAX must be equal; float sums are over non-negative
values, so two orders differ by at most n * 2^-53 of the sum (below 1e-9 for these sizes)."""
import numpy as np
import pytest

from tests.helpers import assert_groups_equal

pytestmark = pytest.mark.gpu

I32, I64, F64, DEC, IPV4 = 1, 2, 4, 17, 8
N = (1 << 20) + 3


def _keys(kind, rng):
    if kind == "range":
        return rng.integers(-9_000, 11_000, N)
    if kind == "outliers":
        k = rng.integers(0, 20_000, N)
        k[rng.random(N) < 0.0003] = (1 << 62) + 5
        k[rng.random(N) < 0.0003] = -(1 << 61)
        return k
    if kind == "sparse":
        return rng.integers(0, 20_000, N) * 0x123456789
    k = rng.integers(0, 20_000, N)  # "hot": a tenth of the rows have one key
    k[rng.random(N) < 0.1] = 77
    return k


def _both(ctx, monkeypatch, kinds, run):
    monkeypatch.setenv("WG_KEY_WINDOW", "1")
    got = run()
    monkeypatch.setenv("WG_KEY_WINDOW", "0")
    assert_groups_equal(got, run(), kinds, rel=1e-9)


@pytest.mark.parametrize("keys", ["range", "outliers", "sparse", "hot"])
@pytest.mark.parametrize("shape", ["groupby", "i64", "f64", "ipv4"])
def test_compiled_shapes(ctx, monkeypatch, shape, keys):
    import wadjet_b200 as wg
    rng = np.random.default_rng(len(keys))
    key, filt = _keys(keys, rng).astype(np.int64), rng.integers(0, 10, N, dtype=np.int32)
    vi, vf = rng.integers(-(1 << 62), 1 << 62, N), rng.random(N)
    C, S, MN, MX = wg.AGG_COUNT, wg.AGG_SUM, wg.AGG_MIN, wg.AGG_MAX

    def run():
        kw = {}
        if shape == "ipv4":
            a = wg.HashAggregate(ctx, [2], [wg.AggColumn(S, 1), wg.AggColumn(C, -1)], ndv_hint=20_000)
            batch = wg.Batch([wg.Column(IPV4, key * 256 + 3), wg.Column(I64, vi)])
            kw["exprs"] = [wg.Expr(I64, [wg.Expr.col(0), wg.Expr.const_i(8), ">>"])]
        else:
            m = 3 if shape == "groupby" else 1
            a = wg.HashAggregate(ctx, [0], [wg.AggColumn(S, 1), wg.AggColumn(C, -1), wg.AggColumn(MN, m),
                                            wg.AggColumn(MX, m)], ndv_hint=20_000)
            cols = [wg.Column(I64, key), wg.Column(F64, vf) if shape == "f64" else wg.Column(I64, vi),
                    wg.Column(I32, filt)]
            if shape == "groupby":
                cols.append(wg.Column(F64, vf))
            batch = wg.Batch(cols)
            kw["filters"] = [(2, wg.OP_LT, 7)]
        dev = wg.DeviceBatch.upload(ctx, batch)
        for _ in range(2):  # the second batch meets a table with its groups
            wg.run_pipeline(ctx, dev, a, device=True, **kw)
        a.finalize()
        assert a.kernel_shape == {"groupby": 2, "i64": 4, "f64": 5, "ipv4": 6}[shape]
        e = a.export()
        a.close()
        dev.close()
        return e

    kinds = {"groupby": ["sum_i", "count", "min_f", "max_f"], "i64": ["sum_i", "count", "min_i", "max_i"],
             "f64": ["sum_f", "count", "min_f", "max_f"], "ipv4": ["sum_i", "count"]}[shape]
    _both(ctx, monkeypatch, kinds, run)


@pytest.mark.parametrize("keys", ["range", "outliers", "sparse", "hot"])
@pytest.mark.parametrize("nulls", [False, True])
@pytest.mark.parametrize("sel", [False, True])
def test_interpreted_plans(ctx, monkeypatch, keys, nulls, sel):
    import wadjet_b200 as wg
    rng = np.random.default_rng(len(keys) + nulls)
    ok = lambda p: rng.random(N) >= p if nulls else None  # noqa: E731
    dec = np.zeros(N, wg.DEC_DTYPE)
    lo = rng.integers(-(1 << 60), 1 << 60, N)
    dec["lo"], dec["hi"] = lo.view(np.uint64), np.where(rng.random(N) < 0.3, rng.integers(-5, 5, N), lo >> 63)
    cols = [wg.Column(I64, _keys(keys, rng).astype(np.int64), ok(0.05)), wg.Column(DEC, dec, ok(0.1), scale=2),
            wg.Column(F64, rng.random(N), ok(0.1)), wg.Column(I32, rng.integers(-50, 50, N, dtype=np.int32), ok(0.1))]
    aggs = [wg.AggColumn(wg.AGG_SUM, 1), wg.AggColumn(wg.AGG_MIN, 1), wg.AggColumn(wg.AGG_MAX, 1),
            wg.AggColumn(wg.AGG_SUM, 4), wg.AggColumn(wg.AGG_MIN, 3), wg.AggColumn(wg.AGG_COUNT, 2)]
    rows = np.flatnonzero(np.random.default_rng(1).random(2 * N) < 0.9).astype(np.uint32)
    rows = rows[rows < N]
    big = np.concatenate([rows, rows])[: N]  # 2^20 entries and more, rows twice
    batch = wg.Batch(cols, sel=np.sort(big) if sel else None)
    expr = wg.Expr(F64, [wg.Expr.col(2), wg.Expr.const_f(3.5), "*"])

    def run():
        a = wg.HashAggregate(ctx, [0], aggs, ndv_hint=20_000)
        wg.run_pipeline(ctx, batch, a, exprs=[expr])
        a.finalize()
        e = a.export()
        a.close()
        return e

    _both(ctx, monkeypatch, ["sum_d", "min_d", "max_d", "sum_f", "min_i", "count"], run)


def test_known_range_of_a_join_payload(ctx, monkeypatch):
    import wadjet_b200 as wg
    rng = np.random.default_rng(3)
    b = 60_000
    join = wg.HashJoin(ctx, 0, 0, payload=[1], build_row_hint=b)
    join.build([wg.Batch([wg.Column(I64, np.arange(b) * 977), wg.Column(I32, (np.arange(b) % 30_011).astype(np.int32) - 7)])])
    batch = wg.Batch([wg.Column(I64, rng.integers(0, b + 5000, N) * 977), wg.Column(I64, rng.integers(0, 1 << 40, N))])

    def run():
        a = wg.HashAggregate(ctx, [2], [wg.AggColumn(wg.AGG_SUM, 1), wg.AggColumn(wg.AGG_COUNT, -1)], ndv_hint=30_011)
        wg.run_pipeline(ctx, batch, a, join=join)
        a.finalize()
        e = a.export()
        a.close()
        return e

    _both(ctx, monkeypatch, ["sum_i", "count"], run)
    join.close()


@pytest.mark.parametrize("left", [4 << 20, 96 << 10])
def test_buffers_kept_for_speed_refuse_nothing(left):
    """Under a budget the window and the result staging give way: another allocation gets the
    window's memory, and a result that its two staging slots do not fit is read in smaller
    chunks, exports and pages alike."""
    import torch
    import wadjet_b200 as wg
    rng = np.random.default_rng(left)
    key = torch.from_numpy(rng.integers(0, 200_000, N)).cuda()
    val = torch.from_numpy(rng.integers(-100, 100, N)).cuda()
    cols = [wg.Column(I64, key), wg.Column(I64, val)]

    def run(ctx):
        a = wg.HashAggregate(ctx, [0], [wg.AggColumn(wg.AGG_SUM, 1), wg.AggColumn(wg.AGG_COUNT, -1)],
                             ndv_hint=200_000)
        wg.run_pipeline(ctx, wg.Batch(cols), a, device=True)
        a.finalize()
        return a

    def pages(a):
        out = []
        while (page := a.next(130_000)) is not None:
            out.append([np.array(v) for v, _ in page])
        return np.stack([np.concatenate(c) for c in zip(*out)])

    with wg.Context(0) as ctx:
        a = run(ctx)
        want, want_pages = a.export(), pages(a)
        a.close()
    budget = 256 << 20
    with wg.Context(0, hbm_budget=budget) as ctx:
        a = run(ctx)
        used = ctx.ledger()["used"]
        ctx.reserve(budget - used + (8 << 20))  # more than is free: the window's memory is given up
        ctx.reserve(budget - ctx.ledger()["used"] - left)
        got, got_pages = a.export(), pages(a)
        assert ctx.ledger()["peak"] <= budget
        a.close()
    assert_groups_equal(got, want, ["sum_i", "count"])
    order = lambda p: p[:, np.argsort(p[0])]
    np.testing.assert_array_equal(order(got_pages), order(want_pages))


def _wide_query(wg, rng):
    """Rows whose 200,000 groups take a key window, and the groups they give."""
    import torch
    key, val = rng.integers(0, 200_000, N), rng.integers(-100, 100, N)
    keep = [torch.from_numpy(key).cuda(), torch.from_numpy(val).cuda()]
    uniq, at = np.unique(key, return_inverse=True)
    want = dict(keys=uniq, i64=np.bincount(at, val).astype(np.int64), count=np.bincount(at))
    return wg.Batch([wg.Column(I64, keep[0]), wg.Column(I64, keep[1])]), keep, want


def _equal(e, want):
    order = np.argsort(e["keys"][0])
    np.testing.assert_array_equal(e["keys"][0][order], want["keys"])
    np.testing.assert_array_equal(e["i64"][0][order], want["i64"])
    np.testing.assert_array_equal(e["count"][1][order], want["count"])


def test_kept_buffers_of_two_threads():
    """One context, two threads with an aggregate each, and a third whose reservations make the
    context give its kept buffers back: a buffer in use stays its user's. A query that another
    thread's reservation leaves no room says so; every other result is exact."""
    import threading
    import wadjet_b200 as wg
    budget = 512 << 20
    with wg.Context(0, hbm_budget=budget) as ctx:
        batch, keep, want = _wide_query(wg, np.random.default_rng(5))
        stop, errors, good = threading.Event(), [], [0, 0]

        def query(i):
            try:
                for _ in range(25):
                    a = wg.HashAggregate(ctx, [0], [wg.AggColumn(wg.AGG_SUM, 1), wg.AggColumn(wg.AGG_COUNT, -1)],
                                         ndv_hint=200_000)
                    try:
                        wg.run_pipeline(ctx, batch, a, device=True)
                        a.finalize()
                        e = a.export()
                    except wg.MemoryExceeded:
                        continue
                    finally:
                        a.close()
                    _equal(e, want)
                    good[i] += 1
            except BaseException as x:  # noqa: BLE001
                errors.append(x)

        def squeeze():
            while not stop.is_set():
                n = budget - ctx.ledger()["used"] + (1 << 20)
                try:
                    ctx.reserve(n)
                    ctx.release(n)
                except wg.MemoryExceeded:
                    pass
                stop.wait(0.002)

        threads = [threading.Thread(target=query, args=(i,)) for i in range(2)]
        third = threading.Thread(target=squeeze)
        for t in threads + [third]:
            t.start()
        for t in threads:
            t.join()
        stop.set()
        third.join()
        assert not errors, errors[0]
        assert sum(good) >= 10
        ctx.synchronize()
        assert ctx.ledger()["peak"] <= budget


def test_a_server_gives_its_slots_buffers_back():
    """What a server's slots keep is charged to the budget they share, and gives way to a
    reservation of the server's context."""
    import wadjet_b200 as wg
    budget = 1 << 30
    with wg.Context(0, hbm_budget=budget) as ctx:
        batch, keep, want = _wide_query(wg, np.random.default_rng(6))
        s = wg.Server(ctx, 2)
        tickets = [s.submit(batch=batch, group_by=[0], aggs=[wg.AggColumn(wg.AGG_SUM, 1), wg.AggColumn(wg.AGG_COUNT, -1)],
                            ndv_hint=200_000) for _ in range(4)]
        for t in tickets:
            n, _ = s.wait(t, timeout=60.0)
            _equal(s.export(t, n), want)
            s.release(t)
        free = budget - ctx.ledger()["used"]
        ctx.reserve(free + (16 << 20))
        ctx.release(free + (16 << 20))
        s.close()
