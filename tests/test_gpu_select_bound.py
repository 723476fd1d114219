"""GPU tests of how much memory the kept Filter and Project plans of many tables
hold together: at most 128 MB of device memory beside the tables, given back with
them, and calls whose plan has been dropped meanwhile give the same rows."""
from __future__ import annotations

import ctypes as C
import gc

import numpy as np
import pytest

from vexq_b200 import abi, plan as P
from vexq_b200.table import HostTable, float_column, int_column

pytestmark = pytest.mark.gpu

ROWS, TABLES, BOUND = 400_000, 9, 128 << 20


def live():
    v = C.c_int64()
    abi.check(abi.load().vexq_debug_live_device_bytes(C.byref(v)))
    return v.value


def test_kept_buffers_are_bounded_over_all_tables(gpu_lib):
    X = gpu_lib
    gc.collect()
    start = live()
    rng = np.random.default_rng(1)
    a, b = rng.integers(0, 100, ROWS), rng.integers(0, 1000, ROWS).astype(float)
    tables = [X.GpuTable(HostTable([int_column("a", a + i), float_column("b", b)], ROWS, 65536)) for i in range(TABLES)]
    base = live()
    preds = [P.col(0) >= 0, P.col(0) >= 2]

    def project(i, pred):
        # eight columns' images and validity: 9 x 8 bytes a row, 29 MB a plan
        exprs = [P.col(0), P.col(1)] + [P.col(1) + float(k) for k in range(6)]
        res = X.GpuProject(tables[i], exprs, predicate=pred).run()
        n, first = res.nrows, res.next()
        res.close()
        return n, [v.values[:40] for v in first.vectors]

    def want(i, least):
        keep = a + i >= least
        cols = [(a + i)[keep], b[keep]] + [b[keep] + float(k) for k in range(6)]
        return int(keep.sum()), [c[:40].tolist() for c in cols]

    for turn in range(2):
        for i in range(TABLES):
            for pred, least in zip(preds, (0, 2)):
                assert project(i, pred) == want(i, least)
                assert live() - base <= BOUND, (turn, i, live() - base)
            assert X.GpuFilter(tables[i], preds[1]).bitmap()[1] == int((a + i >= 2).sum())
    for t in tables:
        t.close()
    assert live() == start
