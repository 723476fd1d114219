"""GPU tests of how a batch divides its classes into units: the register-path
class keeps four units a resident block, whose rows set the rounding of its float
sums, whatever the group tables take."""
from __future__ import annotations

import re

import pytest

from vexq_b200 import datagen as D, plan as P, workloads as W

pytestmark = pytest.mark.gpu


def units(batch):
    return {k: int(v) for k, v in re.findall(r"(\w+_units)=(\d+)", batch.explain())}


def test_register_class_units_do_not_follow_the_tables(gpu_lib):
    X = gpu_lib
    li = X.GpuTable(D.lineitem(3_000_000, seed=2))
    zt = X.GpuTable(D.zipf_groups(400_000, 500, seed=3))
    q1, q6 = X.GpuHashAggregate(li, W.q1_plan()), X.GpuHashAggregate(li, W.q6_plan())
    zipf = X.GpuHashAggregate(zt, P.AggPlan(None, [0], [P.sum_(P.col(1), "s")]))
    alone, mixed = X.GpuBatch([q1, q6]), X.GpuBatch([q1, q6, zipf])
    try:
        # about four units for each of the class's resident blocks, a whole number an SM
        n = units(alone)["regs_units"]
        assert -(-n // 148) % 4 == 0, alone.explain()
        assert units(mixed)["regs_units"] == n
        assert "unit_div=4/2/4" in mixed.explain()
        for a, b in zip(alone.exec(), mixed.exec()):
            assert a.rows() == b.rows()
    finally:
        for x in (alone, mixed, q1, q6, zipf):
            x.close()
