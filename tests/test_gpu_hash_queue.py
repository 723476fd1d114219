"""GPU tests of the hashed GROUP BY's queue of rows that miss their home slot:
tables from one group to nearly a key a row, ragged row counts around a warp's
chunk, filters that keep nothing, a few rows and all, the key equal to the empty
sentinel, every kind of aggregate with NULLs, two-column keys and runs that size
their table from the run before; against the oracle (whole values: its sums are
exact)."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import refcpu as R
from tests.helpers import assert_rows_match
from vexq_b200 import plan as P
from vexq_b200.table import HostTable, date_column, float_column, int_column

pytestmark = pytest.mark.gpu


def table(n, keys, seed, wide):
    rng = np.random.default_rng(seed)
    k = rng.integers(0, keys, n)
    key = np.where(k == 0, -1, k * (1_000_000_007_000 if wide else 4_000_000 // keys) + (k % 3))  # two columns: codes of 4M x 11
    ok = rng.random(n) >= 0.25
    return HostTable([int_column("k", key), date_column("d", (8000 + k % 11).astype(np.int32)), int_column("f", rng.integers(0, 100, n)),
                      float_column("v", rng.integers(-1000, 1001, n).astype(float), ok), float_column("w", rng.integers(0, 9, n).astype(float)),
                      int_column("i", rng.integers(-50, 50, n), ok)], n, 4096)


AGGS = [P.sum_(P.col(3), "s"), P.count_star("n"), P.sum_(P.col(4), "t"), P.avg(P.col(3), "a"), P.min_(P.col(5), "lo"), P.max_(P.col(4), "hi"),
        P.sum_(P.col(5), "si"), P.count(P.col(3), "c"), P.count_distinct(P.col(4), "cd")]


@pytest.mark.parametrize("keep", [0, 3, 100])
@pytest.mark.parametrize("by", [[0], [0, 1]])
@pytest.mark.parametrize("n,keys", [(1, 1), (127, 130), (129, 7), (4_097, 1), (9_000, 40), (50_003, 9_000), (131_000, 120_000)])
def test_matches_the_oracle(gpu_lib, n, keys, by, keep):
    X = gpu_lib
    host = table(n, keys, n + keys, len(by) == 1)
    plan = P.AggPlan(P.col(2) < keep if keep < 100 else None, by, AGGS)
    t = X.GpuTable(host)
    op = X.GpuHashAggregate(t, plan)
    want = R.agg(R.RefTable(host), plan, workers=0).rows()
    try:
        for _ in range(2):
            assert_rows_match(op.run().rows(), want, ordered=True, rtol=0.0)
    finally:
        op.close()
        t.close()
