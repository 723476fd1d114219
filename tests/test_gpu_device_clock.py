"""GPU tests of a run's times by the device clock: positive, the scan within the
run, the run within the host's wall time, on every path that stamps it (merged
in the scan, group tables of both assembly sizes, top-k in place, compacted for
HAVING, a join's waited-for and following builds) and by events on the paths
that do not; and integer-only joins whose scan merges its own partials."""
from __future__ import annotations

import time

import numpy as np
import pytest

from oracle import refcpu as R
from tests.helpers import assert_rows_match
from vexq_b200 import plan as P
from vexq_b200.table import HostTable, float_column, int_column

pytestmark = pytest.mark.gpu

N = 300_000


def items(seed=3):
    rng = np.random.default_rng(seed)
    return HostTable([int_column("k", rng.integers(0, 4, N)), int_column("m", rng.integers(0, 3000, N)), int_column("l", rng.integers(0, 30_000, N)),
                      float_column("v", rng.integers(-999, 1000, N).astype(float)), int_column("fk", rng.integers(0, 50_000, N))], N, 65536)


def orders(dup=1, n=50_000):
    rng = np.random.default_rng(4)
    return HostTable([int_column("k", rng.permutation(np.arange(n) // dup)), int_column("g", rng.integers(0, 6, n)),
                      int_column("w", rng.integers(-9, 10, n))], n, 4096)


S = [P.sum_(P.col(3), "s"), P.count_star("n")]
AGG = {"merged": P.AggPlan(None, [0], S), "merge kernel": P.AggPlan(None, [0], [P.max_(P.col(3), "x")]), "small table": P.AggPlan(None, [1], S),
       "large table": P.AggPlan(None, [2], S), "top-k": P.AggPlan(None, [2], S, order_col=1, descending=True, limit=5),
       "having": P.AggPlan(None, [2], S, order_col=1, descending=True, limit=5, having=P.col(2) > 9)}
V = P.col(3 + 3)
J = {"integer": [P.count_star("n"), P.sum_(P.col(2), "s"), P.min_(P.col(3 + 1), "lo"), P.max_(P.col(2), "hi")], "float": [P.sum_(V, "s"), P.count_star("n")]}


def timed_runs(op, want, runs=3):
    for _ in range(runs):
        t0 = time.perf_counter()
        r = op.run()
        wall = (time.perf_counter() - t0) * 1e3
        assert 0 < r.scan_ms <= r.kernel_ms <= wall, (r.scan_ms, r.kernel_ms, wall)
        assert_rows_match(r.rows(), want, ordered=True, rtol=0.0)


@pytest.mark.parametrize("path", list(AGG))
def test_aggregate_times(gpu_lib, path):
    X = gpu_lib
    host = items()
    t = X.GpuTable(host)
    op = X.GpuHashAggregate(t, AGG[path])
    try:
        timed_runs(op, R.agg(R.RefTable(host), AGG[path], workers=0).rows())
    finally:
        op.close()
        t.close()


@pytest.mark.parametrize("bits", [0, 4])
@pytest.mark.parametrize("dup", [1, 3])
@pytest.mark.parametrize("group", [1, 3 + 1, 0])
@pytest.mark.parametrize("aggs", list(J))
def test_join_times(gpu_lib, aggs, group, dup, bits):
    X = gpu_lib
    o, i = orders(dup), items()
    plan = P.JoinPlan(0, 4, None, P.col(0) < 3, None, [group], J[aggs], radix_bits=bits)
    to, ti = X.GpuTable(o), X.GpuTable(i)
    op = X.GpuParallelHashJoinAggregate(to, ti, plan)
    try:
        timed_runs(op, R.join(R.RefTable(o), R.RefTable(i), plan, workers=0).rows())
    finally:
        op.close()
        to.close()
        ti.close()
