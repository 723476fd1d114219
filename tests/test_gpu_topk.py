"""GPU tests of ORDER BY an aggregate LIMIT k over group tables: limits around
the block select's sizes (256 and 257 take different selects; 4,096 is the
largest), few groups in a large table, ties across the threshold (every tied
group, in insertion order), NULL aggregates (sorted first), ascending and
descending, float and integer sort columns, and more ties than the candidate
buffer holds; against the oracle's ExternalSort + Limit."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import refcpu as R
from tests.helpers import assert_rows_match
from vexq_b200 import plan as P
from vexq_b200.table import HostTable, float_column, int_column

pytestmark = pytest.mark.gpu


def table(n, keys, seed, wide=True, ties=0, nulls=0.0):
    rng = np.random.default_rng(seed)
    k = rng.integers(0, keys, n)
    k[:min(keys, n)] = np.arange(min(keys, n))
    rng.shuffle(k)
    # whole values: the oracle's serial fold is exact too, so its ties are ties here
    v = rng.integers(0, ties, n).astype(float) if ties else rng.integers(-10_000, 10_000, n).astype(float)
    key = k * 1_000_000_007 if wide else k
    return HostTable([int_column("k", key), float_column("v", v, rng.random(n) >= nulls if nulls else None),
                      int_column("i", rng.integers(-50, 50, n))], n, 65536)


AGGS = [P.sum_(P.col(1), "s"), P.count_star("n"), P.max_(P.col(1), "x"), P.avg(P.col(1), "a"), P.sum_(P.col(2), "si")]


@pytest.mark.parametrize("limit", [0, 1, 10, 256, 257, 1000, 4096])
@pytest.mark.parametrize("col,desc", [(1, True), (1, False), (2, True), (3, True), (4, False), (5, True)])
def test_matches_the_oracle(gpu_lib, limit, col, desc):
    X = gpu_lib
    host = table(60_000, 30_000, limit + col, nulls=0.2)
    plan = P.AggPlan(None, [0], AGGS, order_col=col, descending=desc, limit=limit)
    t = X.GpuTable(host)
    op = X.GpuHashAggregate(t, plan)
    want = R.agg(R.RefTable(host), plan, workers=0).rows()
    try:
        for _ in range(2):
            assert_rows_match(op.run().rows(), want, ordered=True, rtol=0.0)
    finally:
        op.close()
        t.close()


@pytest.mark.parametrize("n,keys,ties,limit", [(400_000, 200_000, 1, 10), (100_000, 50_000, 3, 300), (300, 200, 0, 7), (70_000, 66_000, 1, 20)])
def test_ties_and_few_groups(gpu_lib, n, keys, ties, limit):
    """ties=1: every integer-valued sum is 0, all groups tie (200,000 of them
    do not fit the candidate buffer); the first in insertion order win."""
    X = gpu_lib
    for wide in (True, False):
        host = table(n, keys, 5, wide=wide, ties=ties)
        plan = P.AggPlan(None, [0], [P.sum_(P.col(1), "s"), P.count_star("n")], order_col=1, descending=True, limit=limit)
        t = X.GpuTable(host)
        op = X.GpuHashAggregate(t, plan)
        try:
            want = R.agg(R.RefTable(host), plan, workers=0).rows()
            for _ in range(2):
                assert_rows_match(op.run().rows(), want, ordered=True, rtol=0.0)
        finally:
            op.close()
            t.close()
