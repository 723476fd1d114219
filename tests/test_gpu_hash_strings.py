"""GPU tests of a hashed GROUP BY whose keys are all dictionary strings, more
combinations than a dense table takes: groups come in the integer-key path's
insertion order, NULL-keyed groups first (exec/agg_intkey.go:249-255), alone and
in a batch; against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import refcpu as R
from tests.helpers import assert_rows_match
from vexq_b200 import plan as P
from vexq_b200.table import HostTable, float_column, int_column, string_column

pytestmark = pytest.mark.gpu

AGGS = [P.count_star("n"), P.sum_(P.col(3), "s"), P.min_(P.col(4), "lo"), P.avg(P.col(3), "a")]


def table(n, sizes, nulls, seed, spread):
    rng = np.random.default_rng(seed)
    cols = []
    for j, size in enumerate(sizes):
        idx = np.concatenate([rng.permutation(size), rng.integers(0, spread, max(0, n - size))])[:n]
        cols.append(string_column(f"k{j}", idx, [f"{j}_{i}" for i in range(size)], n, 4096, rng.random(n) >= 0.2 if nulls[j] else None))
    while len(cols) < 3:
        cols.append(int_column("pad", np.zeros(n, np.int64)))
    v = rng.integers(-1000, 1001, n).astype(float)
    return HostTable(cols + [float_column("v", v, rng.random(n) >= 0.25), int_column("i", rng.integers(-50, 50, n))], n, 4096)


@pytest.mark.parametrize("n,sizes,nulls,spread", [
    (2_100, (2_100, 2_100), (False, False), 2_100),
    (40_003, (2_100, 2_100), (False, False), 9),
    (40_003, (2_700, 2_100), (True, False), 40),
    (60_001, (2_048, 2_048), (True, True), 2_048),
    (9_000, (400, 400, 60), (True, True, True), 5),
])
def test_matches_the_oracle(gpu_lib, n, sizes, nulls, spread):
    X = gpu_lib
    host = table(n, sizes, nulls, n + sum(nulls), spread)
    plan = P.AggPlan(P.col(4) < 45, list(range(len(sizes))), AGGS)
    t = X.GpuTable(host)
    op = X.GpuHashAggregate(t, plan)
    assert "path=hash" in op.explain()
    want = R.agg(R.RefTable(host), plan, workers=0).rows()
    batch = X.GpuBatch([op])
    try:
        for _ in range(2):
            assert_rows_match(op.run().rows(), want, ordered=True, rtol=0.0)
            assert_rows_match(batch.exec()[0].rows(), want, ordered=True, rtol=0.0)
    finally:
        batch.close()
        op.close()
        t.close()
