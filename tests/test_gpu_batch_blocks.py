"""GPU tests of the pinned blocks the device writes result columns to: above a
size a batch keeps one for every execution and its results copy their rows, and a
block that cannot be pinned is no error."""
from __future__ import annotations

import numpy as np
import pytest

from tests.plan_probe import Probe
from vexq_b200 import plan as P
from vexq_b200.table import HostTable, float_column, int_column

pytestmark = pytest.mark.gpu


def test_large_blocks_are_not_lent(gpu_lib, tmp_path):
    probe = Probe(str(tmp_path))
    mb = 1 << 20
    assert probe.out_pool(4, 24 * mb, 64 * mb) == (3 * 32 * mb, 2)  # pinned by powers of two up to 32 MB
    assert probe.out_pool(4, 96 * mb, 64 * mb) == (96 * mb, 0)
    probe.close()


def test_results_of_a_large_batch_held_over_executions(gpu_lib):
    # three hashed tables of 2^20 slots, three columns each: 75 MB a block
    X = gpu_lib
    n, groups = 500_000, 1_500
    rng = np.random.default_rng(4)
    tables, ops, want = [], [], []
    for i in range(3):
        k = rng.integers(0, groups, n) * 1_000_003_000_017
        v = rng.integers(0, 1000, n).astype(float)
        t = X.GpuTable(HostTable([int_column("k", k), float_column("v", v)], n, 65536))
        tables.append(t)
        ops.append(X.GpuHashAggregate(t, P.AggPlan(None, [0], [P.sum_(P.col(1), "s"), P.count_star("n")])))
        keys, first, inv = np.unique(k, return_index=True, return_inverse=True)
        sums, counts = np.bincount(inv, v), np.bincount(inv)
        want.append([(int(keys[j]), float(sums[j]), int(counts[j])) for j in np.argsort(first)])
    batch = X.GpuBatch(ops)
    held = [batch.exec() for _ in range(4)]
    batch.close()
    for results in held:
        for res, rows in zip(results, want):
            assert [tuple(r) for r in res.rows()] == rows
    for x in ops + tables:
        x.close()


def test_a_block_that_cannot_be_pinned_is_none(gpu_lib, tmp_path):
    # the caller then takes the way that needs no block (2^46 bytes: more than the address space holds)
    probe = Probe(str(tmp_path))
    assert probe.out_pool(2, 1 << 46, 1 << 62) == (0, 0)
    assert probe.out_pool(2, 1 << 20, 1 << 62)[1] == 2
    probe.close()
