"""GPU tests of the float sums' windows where more than 2^31 rows may meet in
one group (a join of repeated keys): the window that leaves room above the
values, chosen by what the keys could emit, and one group that does take 2.3e9
rows of values next to the column's bound. Sums are exact, so they are compared
as such."""
from __future__ import annotations

from fractions import Fraction

import numpy as np
import pytest

from vexq_b200 import plan as P
from vexq_b200.table import HostTable, float_column, int_column

pytestmark = pytest.mark.gpu

GROUPS = 40


def check(X, chain, probes, idle, values):
    """Key 0 has `chain` build rows, all of group 7; keys 1 ... GROUPS - 1 have
    one each, of a group of their own. `idle` probe rows match nothing."""
    bk = np.concatenate([np.zeros(chain, np.int64), np.arange(1, GROUPS)])
    bg = np.concatenate([np.full(chain, 7), (np.arange(1, GROUPS) + 7) % GROUPS])
    pk = np.concatenate([np.zeros(probes, np.int64), np.arange(1, GROUPS), np.full(idle, GROUPS + 5)])
    pv = np.resize(np.asarray(values, float), len(pk))
    tb = X.GpuTable(HostTable([int_column("k", bk), int_column("g", bg)], len(bk), 4096))
    tp = X.GpuTable(HostTable([int_column("k", pk), float_column("v", pv)], len(pk), 4096))
    op = X.GpuParallelHashJoinAggregate(tb, tp, P.JoinPlan(0, 0, None, None, None, [1], [P.sum_(P.col(3), "s"), P.count_star("n"), P.avg(P.col(3), "a")]))
    vals, counts = np.unique(pv[:probes], return_counts=True)
    heavy = float(chain * sum(Fraction(float(v)) * int(n) for v, n in zip(vals, counts)))
    want = {(k + 7) % GROUPS: (float(pv[probes + k - 1]), 1) for k in range(1, GROUPS)}
    want[7] = (heavy, chain * probes)
    try:
        for _ in range(2):
            rows = op.run().rows()
            assert {r[0]: (r[1], r[2]) for r in rows} == want
            assert all(r[3] == r[1] / r[2] for r in rows)
    finally:
        op.close()
        tb.close()
        tp.close()


# at the bound, over 43 binades below it (every bit lies in both windows), of both signs
@pytest.mark.parametrize("values", [[1.9999], [1.9999, 2.0 ** -43, 3.5 * 2.0 ** -42], [-1.9999, 1.75, -2.0 ** -42, 0.0]])
@pytest.mark.parametrize("chain,probes,idle", [(3, 2_000, 0), (2_000, 3, 0), (1_500, 2_001, 0), (20_000, 50, 110_000)])
def test_sums_are_exact_in_either_window(gpu_lib, chain, probes, idle, values):
    check(gpu_lib, chain, probes, idle, values)


def test_a_group_of_more_rows_than_the_narrow_window_holds(gpu_lib):
    # 2.3e9 rows of 3.75: 9.26e18 in units of a digit that holds 2^63 = 9.22e18
    check(gpu_lib, 46_000, 50_000, 0, [3.75])
