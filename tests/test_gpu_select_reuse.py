"""GPU tests of Filter and Project calls that reuse a table's compiled plans and
buffers: the same expression again, other literals, other row ranges, results
of several calls alive at once, and a refill that widens a column's range in
between; each against the oracle."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from oracle import refcpu as R
from tests.helpers import assert_rows_match
from tests.test_gpu_select import nullable_table
from vexq_b200 import plan as P
from vexq_b200.table import HostTable, float_column, int_column

pytestmark = pytest.mark.gpu

A, B, D, S = (P.col(i) for i in range(4))


def project(X, t, pred):
    return X.GpuProject(t, [A, B * 2.0, D, S, P.is_null(B)], predicate=pred).run()


def test_project_results_alive_together(gpu_lib):
    X = gpu_lib
    host = nullable_table(n=30_011)
    t, rt = X.GpuTable(host), R.RefTable(host)
    preds = [A > 10, A > 30, A > 10, A > 49, None, A > 10, P.and_(A < 0, P.in_(S, ["x", "zz"])), A > 10]
    held = [project(X, t, p) for p in preds]
    t_rows = [R.project(rt, [A, B * 2.0, D, S, P.is_null(B)], p).rows() for p in preds]
    t.close()  # results outlive the table and its plans
    for res, want in zip(held, t_rows):
        assert_rows_match(res.rows(), want, ordered=True, rtol=0.0)


@pytest.mark.parametrize("lo,hi", [(0, -1), (1, 30_000), (8, 8), (7, 9), (4095, 4097), (29_999, 30_011), (0, 1)])
def test_bitmap_ranges_on_a_kept_plan(gpu_lib, lo, hi):
    X = gpu_lib
    host = nullable_table(n=30_011)
    t = X.GpuTable(host)
    n = host.nrows if hi < 0 else hi
    for pred in (A > 10, A > 30, A > 10):
        want = np.unpackbits(np.frombuffer(R.filter_bits(R.RefTable(host), pred)[0], dtype=np.uint8), bitorder="little")[lo:n]
        X.GpuFilter(t, pred).bitmap()  # leaves bits of the whole table behind
        bits, cnt = X.GpuFilter(t, pred).bitmap(lo, hi)
        assert cnt == int(want.sum())
        assert bits == np.packbits(want, bitorder="little").tobytes()
    t.close()


def test_a_refill_between_calls(gpu_lib):
    X = gpu_lib
    n = 20_000
    rng = np.random.default_rng(0)
    a, b = rng.integers(0, 10, n), np.round(rng.normal(0, 1, n), 2)
    host = HostTable([int_column("a", a), float_column("b", b)], n, 4096)
    t = X.GpuTable(host)
    op = X.GpuHashAggregate(t, P.AggPlan(P.col(0) < 1000, [], [P.count_star("n")]))
    pred = P.col(0) > 5
    assert X.GpuFilter(t, pred).bitmap()[1] == int((a > 5).sum())
    wide = HostTable([int_column("a", a * 1_000_000_007), float_column("b", b * 1e9)], n, 4096)
    try:
        op.run_host(wide).close()
    except Exception:  # the aggregate plan refuses the wider range; the table is refilled
        pass
    assert X.GpuFilter(t, pred).bitmap()[1] == int((a * 1_000_000_007 > 5).sum())
    got = X.GpuProject(t, [P.col(0) + 1, P.col(1) * 2.0], predicate=pred).run().rows()
    keep = a > 0
    assert [r[0] for r in got] == (a[keep] * 1_000_000_007 + 1).tolist()
    assert [r[1] for r in got] == ((b * 1e9)[keep] * 2.0).tolist()
    op.close()
    t.close()


def test_threads_on_one_table(gpu_lib):
    X = gpu_lib
    host = nullable_table(n=30_011)
    t, rt = X.GpuTable(host), R.RefTable(host)
    want = {k: (R.filter_bits(rt, A > k)[0], R.project(rt, [A, B * 2.0, D, S, P.is_null(B)], A > k).rows()) for k in (5, 25)}
    bad = []

    def work(k):
        for _ in range(20):
            if X.GpuFilter(t, A > k).bitmap()[0] != bytes(want[k][0]):
                bad.append(("bits", k))
            try:
                assert_rows_match(project(X, t, A > k).rows(), want[k][1], ordered=True, rtol=0.0)
            except AssertionError as e:
                bad.append((k, str(e)[:100]))
    th = [threading.Thread(target=work, args=(k,)) for k in (5, 25, 5, 25)]
    [x.start() for x in th]
    [x.join() for x in th]
    t.close()
    assert not bad
