"""What plans compile to, checked without a GPU: the generated kernels are
compiled for sm_100a as on a GPU host and not loaded."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

from tests.plan_probe import Probe, abi, column, lsb
from vexq_b200 import plan as P

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("probe")
    with pytest.MonkeyPatch.context() as m:
        m.setenv("VEXQ_JIT_CACHE", str(tmp / "jit"))
        p = Probe(str(tmp))
        yield p
        p.close()


@pytest.mark.parametrize("nullable", [(False, False), (True, False), (True, True)])
def test_hashed_group_by_of_strings_compiles(probe, nullable):
    # 2,100 x 2,100 codes: more than the 2^22 a dense table takes
    t = probe.table([column(abi.TYPE_STRING, n, 2100) for n in nullable] + [column(abi.TYPE_FLOAT64, True, lo=-9, hi=9)], 100_000)
    text = probe.agg(t, P.AggPlan(None, [0, 1], [P.count_star("n"), P.sum_(P.col(2), "s")]))
    assert "path=hash" in text, text


@pytest.mark.parametrize("join", [False, True])
def test_float_sum_windows_hold_every_row(probe, join):
    """A sum's top digit takes up to 2^32 a row into a signed 64-bit counter where
    the window ends with the values: 2^31 rows of one group."""
    def window(nrows):
        t = probe.table([column(abi.TYPE_INT64, lo=0, hi=99), column(abi.TYPE_FLOAT64, lo=0, hi=1.9999)], nrows)
        if join:
            b = probe.table([column(abi.TYPE_INT64, lo=0, hi=99), column(abi.TYPE_INT64, lo=0, hi=99)], 100)
            text = probe.join(b, t, P.JoinPlan(0, 0, None, None, None, [1], [P.sum_(P.col(3), "s")]))
        else:
            text = probe.agg(t, P.AggPlan(None, [0], [P.sum_(P.col(1), "s")]))
        return max(lsb(text)), text  # |x| < 2: the value's top bit weighs 2^0

    for nrows in (1_000, 2 ** 31, 2 ** 31 + 1, 2 ** 32 - 2, 2 ** 33):
        bottom, text = window(nrows)
        top_digit = 2.0 ** (1 - bottom - 96)  # the most a row adds to the counter that weighs 2^(bottom + 96)
        assert top_digit * nrows <= 2.0 ** 63, (nrows, text)
        assert 1 - bottom <= 128 and bottom <= 1 - 97, (nrows, text)  # the window holds the values, 97 bits of them or more


@pytest.mark.parametrize("block", [64, 128, 256, 384, 512])
@pytest.mark.parametrize("shape", ["by_key", "by_date", "registers"])
def test_join_probes_compile_at_every_block_size(probe, monkeypatch, block, shape):
    # the probe's queues are in static shared memory, 48 KB a block at most
    monkeypatch.setenv("VEXQ_TUNE", f"block={block} async=2")
    b = probe.table([column(abi.TYPE_INT64, lo=0, hi=99_999), column(abi.TYPE_DATE, lo=8000, hi=9000), column(abi.TYPE_INT64, lo=0, hi=4)], 100_000)
    t = probe.table([column(abi.TYPE_INT64, lo=0, hi=99_999), column(abi.TYPE_FLOAT64, True, lo=-9, hi=9), column(abi.TYPE_INT64, lo=0, hi=9)], 400_000)
    by = {"by_key": 0, "by_date": 1, "registers": 2}[shape]
    text = probe.join(b, t, P.JoinPlan(0, 0, None, P.col(2) < 3, None, [by], [P.sum_(P.col(4), "s"), P.count_star("n")]))
    assert text.startswith("lsb="), text


def test_a_kept_filter_plan_is_keyed_by_its_expression(probe):
    t = probe.table([column(abi.TYPE_INT64, lo=0, hi=99), column(abi.TYPE_DATE, lo=8000, hi=9000)], 100_000)
    number, date = P.col(0) < 7, P.col(1) < P.lit("1994-01-01")
    assert [n.kind for n in P.predicate_arrays(number)[0].nodes] == [abi.E_COLUMN, abi.E_LITERAL, abi.E_BINARY]
    # lit_str is read of STRING literals only: a caller leaves it unset elsewhere
    key = probe.filter_key(t, number)
    assert all(probe.filter_key(t, number, {i: b"stray"}) == key for i in range(3))
    assert probe.filter_key(t, date, {0: b"stray"}) == probe.filter_key(t, date)
    keys = [probe.filter_key(t, p) for p in (number, P.col(0) < 8, P.col(0) <= 7, date, P.col(1) < P.lit("1994-01-02"))]
    assert len(set(keys)) == len(keys)


@pytest.mark.parametrize("tune,places", [("", 2), ("staged=1", 3)])
def test_a_hashed_kernel_holds_its_update_twice(probe, monkeypatch, tune, places):
    # where rows lie and out of the queue; a third copy for the queue's rest was
    # a quarter of the plan's compile time (the staged loop has no step for it)
    monkeypatch.setenv("VEXQ_TUNE", tune)
    t = probe.table([column(abi.TYPE_INT64, lo=-2 ** 62, hi=2 ** 62), column(abi.TYPE_FLOAT64, True, lo=-9, hi=9)], 100_000)
    plan = P.AggPlan(P.col(1) < 5.0, [0], [P.sum_(P.col(1), "s"), P.count_star("n")])
    assert f"warp_sums={places} " in probe.agg(t, plan)
    assert f"warp_sums={places} " in probe.agg_wide(t, plan)


def test_float_min_max_plans_stay_in_their_arrays(tmp_path):
    # in a process of its own whose allocator checks every block it frees
    code = f"""
from tests.plan_probe import Probe, abi, column
from vexq_b200 import plan as P
probe = Probe({str(tmp_path)!r})
cols = [column(abi.TYPE_INT64, lo=0, hi=999)] + [column(abi.TYPE_FLOAT64, lo=-9, hi=9) for _ in range(6)]
t = probe.table(cols, 100_000)
for k in range(1, 7):
    aggs = [f(P.col(1 + i), f"a{{i}}{{f.__name__}}") for i in range(k) for f in (P.min_, P.max_)]
    assert "path=dense" in probe.agg(t, P.AggPlan(None, [0], aggs))
    assert "path=dense" in probe.agg(t, P.AggPlan(None, [0], aggs + [P.sum_(P.col(1), "s")]))
print("fine")
"""
    env = dict(os.environ, VEXQ_JIT_CACHE=str(tmp_path / "jit"), LD_PRELOAD="libc_malloc_debug.so.0", MALLOC_CHECK_="3")
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, cwd=ROOT)
    assert r.returncode == 0 and "fine" in r.stdout, (r.returncode, r.stderr[-500:])
