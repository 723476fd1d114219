"""GPU tests of COUNT(DISTINCT) under the staged scan loop, whose units are tiles
of several chunks: its set is sized by the tiles' rows; against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import refcpu as R
from tests.helpers import assert_rows_match
from vexq_b200 import plan as P
from vexq_b200.table import HostTable, int_column

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups", [3, 500, 1_000_000_007])
def test_a_value_a_row(gpu_lib, monkeypatch, groups):
    X = gpu_lib
    n = 50_003
    rng = np.random.default_rng(groups)
    g = rng.integers(0, 3, n) if groups == 3 else rng.integers(0, 500, n) * (groups // 500)
    host = HostTable([int_column("g", g), int_column("v", np.arange(n))], n, 4096)
    plan = P.AggPlan(None, [0], [P.count_distinct(P.col(1), "d"), P.count_star("n")])
    monkeypatch.setenv("VEXQ_TUNE", "staged=1")
    t = X.GpuTable(host)
    op = X.GpuHashAggregate(t, plan)
    try:
        for _ in range(2):
            assert_rows_match(op.run().rows(), R.agg(R.RefTable(host), plan, workers=0).rows(), ordered=True, rtol=0.0)
    finally:
        op.close()
        t.close()
