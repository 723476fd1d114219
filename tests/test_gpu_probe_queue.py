"""GPU tests of the join probe's queue of matched rows (a probe filter and few
groups): filters that keep nothing, a few rows, about the count at which a chunk
folds its matches where they lie, and all of them; dense and sparse stretches in
turn; ragged row counts; repeated and NULL keys; a residual over both sides;
against the oracle. The values are whole, so the oracle's sums are exact."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import refcpu as R
from tests.helpers import assert_rows_match
from vexq_b200 import plan as P
from vexq_b200.table import HostTable, bool_column, float_column, int_column

pytestmark = pytest.mark.gpu

NB = 5  # build columns before the probe's in the joined row


def tables(nb, n, seed, keep, dup, nulls):
    rng = np.random.default_rng(seed)
    keys = np.arange(nb) // dup * 3
    some = (lambda m: rng.random(m) >= 0.2) if nulls else (lambda m: None)
    build = HostTable([int_column("k", rng.permutation(keys), some(nb)), int_column("g", rng.integers(0, 5, nb), some(nb)),
                       int_column("w", rng.integers(-9, 10, nb)), float_column("x", rng.integers(-99, 100, nb).astype(float), some(nb)),
                       bool_column("b", rng.random(nb) < 0.5, some(nb))], nb, 4096)
    # stretches of 1,000 rows: as asked, and every third of them the other way
    f = rng.random(n) < np.where(np.arange(n) // 1000 % 3 == 2, 1.0 - keep, keep)
    probe = HostTable([int_column("fk", rng.integers(0, max(nb // dup * 3, 1), n) // 3 * 3, some(n)), int_column("f", f.astype(np.int64)),
                       float_column("v", rng.integers(-1000, 1001, n).astype(float), some(n)), bool_column("c", rng.random(n) < 0.5, some(n)),
                       int_column("i", rng.integers(-50, 50, n))], n, 4096)
    return build, probe


@pytest.mark.parametrize("few", [False, True])  # few accumulators: the loop that prefetches into registers
@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("nb,n,dup,nulls", [(1000, 1, 1, False), (1000, 33, 1, True), (3000, 50_001, 1, False), (3000, 50_001, 3, True),
                                            (60_000, 130_007, 1, True)])
@pytest.mark.parametrize("keep", [0.0, 0.03, 0.6, 0.66, 1.0])
def test_matches_the_oracle(gpu_lib, keep, nb, n, dup, nulls, residual, few):
    X = gpu_lib
    build, probe = tables(nb, n, n + dup, keep, dup, nulls)
    v, c, i = P.col(NB + 2), P.col(NB + 3), P.col(NB + 4)
    aggs = [P.count_star("n"), P.sum_(v, "s"), P.sum_(P.col(2) * i, "p"), P.min_(P.col(3), "lo"), P.max_(i, "hi"), P.avg(v, "a"),
            P.count(P.col(4), "b"), P.count(c, "c")]
    plan = P.JoinPlan(0, 0, None, P.col(1) == 1, (P.col(3) < v) if residual else None, [1], aggs[:2] if few else aggs, radix_bits=0)
    tb, tp = X.GpuTable(build), X.GpuTable(probe)
    op = X.GpuParallelHashJoinAggregate(tb, tp, plan)
    want = R.join(R.RefTable(build), R.RefTable(probe), plan, workers=0).rows()
    try:
        for _ in range(2):
            assert_rows_match(op.run().rows(), want, ordered=True, rtol=0.0)
    finally:
        op.close()
        tb.close()
        tp.close()
