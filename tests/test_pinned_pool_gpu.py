"""GPU test of the pinned-block pool: plans made, run and dropped by several
threads at once, each result read after its plan is gone and after other plans
have taken blocks back from the pool, keeps its own rows."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from vexq_b200 import plan as P
from vexq_b200.table import HostTable, float_column, int_column

pytestmark = pytest.mark.gpu


def test_results_keep_their_blocks(gpu_lib):
    X = gpu_lib
    bad = []

    def work(w):
        rng = np.random.default_rng(w)
        for k in range(8):
            n, groups = int(rng.integers(1_000, 40_000)), int(rng.integers(20, 400))
            g = rng.integers(0, groups, n)
            v = rng.integers(0, 1000, n).astype(float)
            t = X.GpuTable(HostTable([int_column("g", g), float_column("v", v)], n, 4096))
            held = []
            for _ in range(4):
                op = X.GpuHashAggregate(t, P.AggPlan(None, [0], [P.sum_(P.col(1), "s"), P.count_star("n")]))
                held.append(op.run())
                held.append(X.GpuProject(t, [P.col(0), P.col(1) + 1.0], predicate=P.col(0) < 5).run())
                op.close()
            t.close()
            want = {int(x): (float(v[g == x].sum()), int((g == x).sum())) for x in np.unique(g)}
            rows = list(zip(g[g < 5].tolist(), (v[g < 5] + 1.0).tolist()))
            for i, r in enumerate(held):
                if i % 2 == 0 and {a: (s, c) for a, s, c in r.rows()} != want:
                    bad.append((w, k, i))
                if i % 2 == 1 and [tuple(x) for x in r.rows()] != rows:
                    bad.append((w, k, i))
    th = [threading.Thread(target=work, args=(w,)) for w in range(4)]
    [x.start() for x in th]
    [x.join() for x in th]
    assert not bad
