"""GPU tests of the dense path's shared-memory group cache: limb sums at their
widest (every mantissa bit set, values of the bound's own binade, all rows of a
block in one group, so limbs are normalised many times), mixed signs and
magnitudes, NaN, integer extremes, the cache's edges (the last
code has an entry of its own; codes past the cache go to the global table).
Float sums must equal the exact sum's double bit for bit."""
from __future__ import annotations

import math

import numpy as np
import pytest

from vexq_b200 import plan as P
from vexq_b200.table import HostTable, float_column, int_column

pytestmark = pytest.mark.gpu


def values(kind, n, rng):
    if kind == "top":         # 0 <= x < 2^17, every mantissa bit set: the largest limbs
        return np.full(n, np.nextafter(2.0 ** 17, 0))
    if kind == "positive":    # six decades, all bits random
        return rng.random(n) * 10.0 ** rng.integers(-3, 4, n)
    if kind == "signed":
        return (rng.random(n) - 0.5) * 10.0 ** rng.integers(-20, 16, n)
    if kind == "negative":
        return -rng.random(n) * 1e5
    x = rng.normal(0, 100, n)
    x[rng.integers(0, n, 50)] = np.nan  # (a column holding an infinity has no range and its SUM is refused)
    return x


@pytest.mark.parametrize("kind", ["top", "positive", "signed", "negative", "nan"])
@pytest.mark.parametrize("n,groups,hot", [(3_000_001, 17, 0.99), (300_007, 1755, 0.3), (320_000, 2600, 0.1), (40_003, 40, 0.5),
                                          (1_000, 20, 0.0)])
def test_sums_are_exact(gpu_lib, kind, n, groups, hot):
    X = gpu_lib
    rng = np.random.default_rng(groups)
    g = rng.integers(0, groups, n)
    g[rng.random(n) < hot] = groups - 1  # the last code is the hot one
    g[:groups] = np.arange(groups)
    valid = rng.random(n) >= 0.05
    valid[0] = True
    x = values(kind, n, rng)
    i = rng.integers(-(1 << 62), 1 << 62, n)
    host = HostTable([int_column("g", g, valid), float_column("x", x), int_column("i", i)], n, 65536)
    t = X.GpuTable(host)
    op = X.GpuHashAggregate(t, P.AggPlan(None, [0], [P.sum_(P.col(1), "s"), P.count_star("n"), P.min_(P.col(1), "mn"), P.max_(P.col(1), "mx"),
                                                     P.sum_(P.col(2), "si"), P.min_(P.col(2), "mi"), P.max_(P.col(2), "xi")]))
    try:
        assert "path=dense" in op.explain() and "smem_groups=0" not in op.explain()
        rows = op.run().rows()
    finally:
        op.close()
        t.close()
    key = np.where(valid, g, -1)
    order = np.argsort(key, kind="stable")
    starts = np.flatnonzero(np.r_[True, key[order][1:] != key[order][:-1]])
    want = {}
    for a, b in zip(starts, np.r_[starts[1:], n]):
        sel = order[a:b]
        v = x[sel]
        fin = v[~np.isnan(v)]
        s = math.nan if np.isnan(v).any() else math.fsum(v)
        want[key[sel[0]]] = (order[a], s, b - a, fin.min(), fin.max(), int(i[sel].astype(np.uint64).sum(dtype=np.uint64).astype(np.int64)),
                             int(i[sel].min()), int(i[sel].max()))
    assert [(-1 if r[0] is None else r[0]) for r in rows] == [k for k, _ in sorted(want.items(), key=lambda kv: kv[1][0])]
    for r in rows:
        _, s, cnt, mn, mx, si, mi, xi = want[-1 if r[0] is None else r[0]]
        assert r[2] == cnt and (r[3], r[4], r[5], r[6], r[7]) == (mn, mx, si, mi, xi), r
        if kind == "signed":  # values below 2^-45 of the bound lose bits in the exact window
            assert abs(r[1] - s) <= 2.0 ** -45 * 2.0 ** -44 * np.abs(x).max() * cnt + 1e-300 + abs(s) * 2.0 ** -53, (r, s)
        else:
            assert r[1] == s or (math.isnan(s) and math.isnan(r[1])), (r, s)
