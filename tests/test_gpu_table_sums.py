"""GPU tests of group tables' exact float sums over the whole window (values from
the largest's binade down to the last one kept exactly: 2^-75 of it in a hashed
table, 2^-44 in the block's group cache) and of hashed tables' first-row order,
with the key equal to the empty sentinel among the groups: against exact sums
rounded once, group by group in first-occurrence order."""
from __future__ import annotations

from fractions import Fraction

import numpy as np
import pytest

from vexq_b200 import plan as P
from vexq_b200.table import HostTable, float_column, int_column

pytestmark = pytest.mark.gpu


def values(n, down, signed, seed):
    rng = np.random.default_rng(seed)
    m = np.ldexp(rng.integers(2**52, 2**53, n).astype(float), -53)  # every mantissa bit in use, [0.5, 1)
    v = np.ldexp(m, -rng.integers(0, down + 1, n))
    v[0] = m[0]
    return v * rng.choice([-1.0, 1.0], n) if signed else v


@pytest.mark.parametrize("signed", [False, True])
@pytest.mark.parametrize("n,groups", [(1, 1), (33, 5), (5_000, 700), (70_001, 30_000), (200_000, 12)])
@pytest.mark.parametrize("kind", ["hash", "dense"])
def test_sums_over_the_window(gpu_lib, kind, n, groups, signed):
    X = gpu_lib
    rng = np.random.default_rng(n + groups)
    g = rng.integers(0, groups, n)
    # wide keys, one of them -1 (all bits set); or codes too many for the register path, whose sums are not these
    k = np.where(g == 0, -1, g * 1_000_003_000_017) if kind == "hash" else g * (499 if groups < 1000 else 1)
    v = values(n, 75 if kind == "hash" else 44, signed, n)
    host = HostTable([int_column("k", k), float_column("v", v)], n, 4096)
    plan = P.AggPlan(None, [0], [P.sum_(P.col(1), "s"), P.count_star("n")])
    t = X.GpuTable(host)
    op = X.GpuHashAggregate(t, plan)
    want, cnt = {}, {}
    for key, x in zip(k.tolist(), v.tolist()):
        want[key] = want.get(key, Fraction(0)) + Fraction(x)
        cnt[key] = cnt.get(key, 0) + 1
    try:
        for _ in range(2):
            rows = op.run().rows()
            assert [tuple(r) for r in rows] == [(key, float(s), cnt[key]) for key, s in want.items()]
    finally:
        op.close()
        t.close()
