"""GPU tests of the end of a device-assembled result by the device clock: when
the whole cluster has written its columns. Its 256 warps take the columns in
turn, so of 32 columns the first warp writes the first only, the key, in about
half the time of an average; of 33 it writes all in turn. The time behind the
scan must not be shorter for the one than for the other."""
from __future__ import annotations

import numpy as np
import pytest

from vexq_b200 import plan as P
from vexq_b200.table import HostTable, float_column, int_column

pytestmark = pytest.mark.gpu


def test_the_slowest_column_is_in_the_kernel_time(gpu_lib):
    X = gpu_lib
    n, rng = 40_000, np.random.default_rng(0)
    cols = [int_column("g", rng.integers(0, 4_000, n))] + [float_column(f"v{i}", rng.normal(0, 1, n)) for i in range(15)]
    t = X.GpuTable(HostTable(cols, n, 65536))
    behind = {}
    for columns in (32, 33):
        op = X.GpuHashAggregate(t, P.AggPlan(None, [0], [P.avg(P.col(1 + i % 15), f"a{i}") for i in range(columns - 1)]))
        runs = []
        for _ in range(30):
            r = op.run()
            runs.append(r.kernel_ms - r.scan_ms)
            r.close()
        behind[columns] = min(runs)
        op.close()
    t.close()
    assert behind[32] > 0.8 * behind[33], behind
