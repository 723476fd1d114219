"""GPU tests of the scan's end by the device clock: when every warp of its last
block is through, not the first. One probe row in the last warp's rows of the
only block has a chain of build rows that outlasts all else of the run."""
from __future__ import annotations

import numpy as np
import pytest

from vexq_b200 import plan as P
from vexq_b200.table import HostTable, float_column, int_column

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("aggs", ["count", "float sum"])
def test_the_last_warp_is_in_the_scan_time(gpu_lib, aggs):
    X = gpu_lib
    chain, probes = 30_000, 1_024  # 1,024 rows: one block of eight warps
    bk = np.concatenate([np.arange(1, 100), np.zeros(chain, np.int64)])
    pk = np.full(probes, 10_000)  # matches nothing
    pk[1_000] = 0
    build = X.GpuTable(HostTable([int_column("k", bk), int_column("g", np.arange(len(bk)) % 40)], len(bk), 65536))
    probe = X.GpuTable(HostTable([int_column("k", pk), float_column("v", np.full(probes, 0.5))], probes, 65536))
    out = [P.count_star("n")] + ([P.sum_(P.col(3), "s")] if aggs == "float sum" else [])
    op = X.GpuParallelHashJoinAggregate(build, probe, P.JoinPlan(0, 0, None, None, None, [1], out))
    try:
        assert "path=dense" in op.explain()
        for _ in range(3):
            r = op.run()
            assert sum(row[1] for row in r.rows()) == chain
            # the build, the table's init and the results take well under a
            # millisecond; 30,000 dependent steps of one warp take several
            assert r.kernel_ms > 2.0
            assert r.scan_ms > 0.5 * r.kernel_ms, (r.scan_ms, r.kernel_ms)
    finally:
        op.close()
        build.close()
        probe.close()
