"""GPU tests of result columns assembled on the device (group tables without
HAVING or ORDER BY): insertion order, NULL-keyed groups first on string keys,
every output type and width, sizes around the 32-row words, the 1,024-row
batches and the table size up to which one cluster writes the columns, against
the oracle; and results that outlive later runs of their plan."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import refcpu as R
from tests.helpers import assert_float_vs_exact, assert_rows_match
from vexq_b200 import plan as P
from vexq_b200.table import HostTable, bool_column, date_column, float_column, int_column, string_column

pytestmark = pytest.mark.gpu


def table(n, card, seed, nulls, rg=4096):
    rng = np.random.default_rng(seed)
    g = rng.integers(0, card, n)
    g[:min(card, n)] = np.arange(min(card, n))
    rng.shuffle(g)

    def valid(p):
        return (rng.random(n) >= p) if nulls else None
    return HostTable([
        string_column("s", g, [f"key-{i}" for i in range(card)], n, rg, valid(0.05)),
        string_column("t", rng.integers(0, 3, n), ["", "x", "yy"], n, rg, valid(0.2)),
        int_column("k", (rng.integers(0, 1 << 40, card))[g]),
        int_column("i", g - 7, valid(0.1)),
        date_column("d", 9000 + rng.integers(0, 5, n), valid(0.3)),
        bool_column("b", rng.integers(0, 2, n), valid(0.1)),
        float_column("v", np.round(rng.normal(0, 1000, n), 2), valid(0.4)),
    ], n, rg)


S, T, K, I, D, B, V = (P.col(i) for i in range(7))
AGGS = [P.count_star("n"), P.count(V, "c"), P.sum_(V, "sv"), P.avg(V, "av"), P.min_(V, "mn"), P.max_(V, "mx"), P.sum_(I, "si"),
        P.min_(D, "md"), P.max_(B, "mb"), P.avg(I, "ai")]


def check(X, host, op, plan, rgs=0, rge=-1):
    ref = R.agg(R.RefTable(host), plan, workers=0, rg_start=rgs, rg_end=rge)
    got = op.run(rgs, rge).rows()
    assert_rows_match(got, ref.rows(), ordered=True, rtol=1e-11)
    assert_float_vs_exact(got, ref, exact_tol=1e-15, rtol=1e-11)


@pytest.mark.parametrize("nulls", [False, True])
@pytest.mark.parametrize("keys,card", [([0], 31), ([0], 32), ([0], 1023), ([0], 1025), ([0, 1], 40), ([1, 4, 5], 20), ([3], 4095),
                                       ([3], 4200), ([0, 3], 300), ([2], 5000)])
def test_groups_match_the_oracle(gpu_lib, keys, card, nulls):
    X = gpu_lib
    host = table(20_003, card, card + nulls, nulls)
    plan = P.AggPlan(None, keys, AGGS)
    t = X.GpuTable(host)
    op = X.GpuHashAggregate(t, plan)
    try:
        if "path=regs" in op.explain():
            pytest.skip("few groups: the register path")
        check(X, host, op, plan)
        check(X, host, op, plan)          # a hash table is sized from the first run
        check(X, host, op, plan, 1, 3)    # a range of row groups, then all again
        check(X, host, op, plan)
    finally:
        op.close()
        t.close()


def test_predicate_limit_and_no_groups(gpu_lib):
    X = gpu_lib
    host = table(9_000, 500, 3, True)
    t = X.GpuTable(host)
    for pred, limit in ((V > 100.0, -1), (V > 100.0, 13), (V > 100.0, 0), (V > 1e9, -1), (None, 1030)):
        plan = P.AggPlan(pred, [0, 1], AGGS, limit=limit)
        op = X.GpuHashAggregate(t, plan)
        try:
            check(X, host, op, plan)
        finally:
            op.close()
    t.close()


def test_results_outlive_later_runs_and_their_plan(gpu_lib):
    """Five results of one plan alive at once, over different row groups, and
    five batch executions: each keeps its own rows."""
    X = gpu_lib
    host = table(5 * 4096, 300, 9, True)
    t = X.GpuTable(host)
    plan = P.AggPlan(None, [0], AGGS)
    op = X.GpuHashAggregate(t, plan)
    refs = [R.agg(R.RefTable(host), plan, workers=0, rg_start=r, rg_end=r + 1).rows() for r in range(5)]
    held = [op.run(r, r + 1) for r in range(5)]
    b = X.GpuBatch([op])
    batches = [b.exec()[0] for _ in range(5)]
    whole = R.agg(R.RefTable(host), plan, workers=0).rows()
    b.close()
    op.close()
    t.close()
    for res, ref in zip(held, refs):
        assert_rows_match(res.rows(), ref, ordered=True, rtol=1e-11)
    for res in batches:
        assert_rows_match(res.rows(), whole, ordered=True, rtol=1e-11)


def test_more_groups_than_the_last_run(gpu_lib):
    """A hash table over 65,536 slots: the block is sized from the last run's
    groups, and a run with more writes them again into a larger one."""
    X = gpu_lib
    n = 300_000
    rng = np.random.default_rng(1)
    keys = rng.permutation(np.arange(n, dtype=np.int64) * 7_000_003)
    keys[:65536] = keys[rng.integers(0, 100, 65536)]
    host = HostTable([int_column("k", keys), float_column("v", np.round(rng.normal(0, 10, n), 1))], n, 65536)
    t = X.GpuTable(host)
    plan = P.AggPlan(None, [0], [P.sum_(P.col(1), "s"), P.count_star("n")])
    op = X.GpuHashAggregate(t, plan)
    try:
        for rgs, rge in ((0, 1), (0, 2), (0, -1), (0, 1), (0, -1)):
            check(X, host, op, plan, rgs, rge)
    finally:
        op.close()
        t.close()


def test_having_set_after_the_batch_was_made(gpu_lib):
    X = gpu_lib
    from vexq_b200 import abi
    host = table(12_000, 200, 5, False)
    t = X.GpuTable(host)
    plan = P.AggPlan(None, [0], [P.count_star("n"), P.sum_(V, "s")])
    op = X.GpuHashAggregate(t, plan)
    b = X.GpuBatch([op])
    whole = b.exec()[0].rows()
    having = P.having_arrays(P.col(1) > 60)
    _, nodes, nn, ch, nc, root, visible = having
    abi.check(abi.load().vexq_plan_set_having(op.h, nodes, nn, ch, nc, root, visible))
    assert b.exec()[0].rows() == [r for r in whole if r[1] > 60]
    abi.check(abi.load().vexq_plan_set_having(op.h, nodes, nn, ch, nc, -1, -1))
    assert b.exec()[0].rows() == whole
    b.close()
    op.close()
    t.close()
