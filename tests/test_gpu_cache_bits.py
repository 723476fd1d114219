"""GPU tests that a dense group table's SUM has the same bits whether or not a
group has an entry in the block's cache: values far below the column's bound,
cut to whole units of 2^(e - 97) (|v| < 2^e) in the cache and beside it, for
every cache size, alone and in a batch."""
from __future__ import annotations

from fractions import Fraction

import numpy as np
import pytest

from vexq_b200 import plan as P
from vexq_b200.table import HostTable, float_column, int_column

pytestmark = pytest.mark.gpu

AGGS = [P.sum_(P.col(1), "s"), P.count_star("n"), P.avg(P.col(1), "a")]


@pytest.mark.parametrize("signed", [False, True])
@pytest.mark.parametrize("down", [45, 60, 96])
@pytest.mark.parametrize("rows,groups", [(9_001, 17), (60_000, 20_000)])
def test_same_bits_for_every_cache_size(gpu_lib, monkeypatch, rows, groups, down, signed):
    X = gpu_lib
    rng = np.random.default_rng(rows + down)
    v = np.ldexp(rng.integers(2**52, 2**53, rows).astype(float), -53 - down)
    if signed:
        v *= rng.choice([-1.0, 1.0], rows)
    v[0] = 1.0  # the bound: |v| < 2^1, units of 2^-96
    k = rng.integers(0, groups, rows)
    want = {}
    for key, x in zip(k.tolist(), v.tolist()):
        units = int(abs(Fraction(x)) * 2**96) * (1 if x > 0 else -1)
        s, n = want.get(key, (0, 0))
        want[key] = (s + units, n + 1)
    rows_want = [(key, float(Fraction(s, 2**96)), n, float(Fraction(s, 2**96)) / n) for key, (s, n) in want.items()]
    t = X.GpuTable(HostTable([int_column("k", k), float_column("v", v)], rows, 4096))
    ops = []
    try:
        for kb in (None, 0, 1, 48, 96, 190):
            if kb is not None:
                monkeypatch.setenv("VEXQ_TUNE", f"cache_kb={kb}")
            ops.append(X.GpuHashAggregate(t, P.AggPlan(None, [0], AGGS)))
            assert "path=dense" in ops[-1].explain()
            assert [tuple(r) for r in ops[-1].run().rows()] == rows_want, kb
        monkeypatch.delenv("VEXQ_TUNE")
        batch = X.GpuBatch(ops[:1])
        assert [tuple(r) for r in batch.exec()[0].rows()] == rows_want
        batch.close()
    finally:
        for op in ops:
            op.close()
        t.close()
