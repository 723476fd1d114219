"""GPU tests of the kernels for group tables of 2^31 - 1 slots or more (a slot
and a sign do not fit a word), on tables of ordinary size: a hashed GROUP BY and
joins whose matches are queued, against the same plans' ordinary kernels and the
oracle."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import refcpu as R
from tests.helpers import assert_rows_match
from tests.plan_probe import Probe
from vexq_b200 import plan as P
from vexq_b200.table import HostTable, float_column, int_column

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def probe(gpu_lib, tmp_path_factory):
    p = Probe(str(tmp_path_factory.mktemp("probe")))
    yield p
    p.close()


def check(op, probe, want):
    try:
        assert_rows_match(op.run().rows(), want, ordered=True, rtol=0.0)
        probe.widen(op)
        for _ in range(2):
            assert_rows_match(op.run().rows(), want, ordered=True, rtol=0.0)
    finally:
        op.close()


@pytest.mark.parametrize("n,keys", [(1, 1), (129, 7), (40_003, 9_000)])
def test_hashed_group_by(gpu_lib, probe, n, keys):
    X = gpu_lib
    rng = np.random.default_rng(n)
    k = rng.integers(0, keys, n)
    host = HostTable([int_column("k", np.where(k == 0, -1, k * 1_000_000_007_000)),
                      float_column("v", rng.integers(-1000, 1001, n).astype(float), rng.random(n) >= 0.2)], n, 4096)
    plan = P.AggPlan(None, [0], [P.sum_(P.col(1), "s"), P.count_star("n"), P.avg(P.col(1), "a")])
    t = X.GpuTable(host)
    check(X.GpuHashAggregate(t, plan), probe, R.agg(R.RefTable(host), plan, workers=0).rows())
    t.close()


@pytest.mark.parametrize("by", [0, 1])
@pytest.mark.parametrize("dup", [1, 3])
def test_join(gpu_lib, probe, dup, by):
    X = gpu_lib
    rng = np.random.default_rng(dup)
    nb, n = 6_000, 30_001
    b = HostTable([int_column("k", rng.permutation(np.arange(nb) // dup)), int_column("g", rng.integers(0, 500, nb))], nb, 4096)
    p = HostTable([int_column("k", rng.integers(0, nb, n)), float_column("v", rng.integers(-1000, 1001, n).astype(float))], n, 4096)
    plan = P.JoinPlan(0, 0, None, P.col(1) < 500.0, None, [by], [P.sum_(P.col(3), "s"), P.count_star("n")])
    tb, tp = X.GpuTable(b), X.GpuTable(p)
    check(X.GpuParallelHashJoinAggregate(tb, tp, plan), probe, R.join(R.RefTable(b), R.RefTable(p), plan, workers=0).rows())
    tb.close()
    tp.close()
