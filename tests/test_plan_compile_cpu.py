"""What plans compile to, checked without a GPU: the generated kernels are
compiled for sm_100a as on a GPU host and not loaded."""
from __future__ import annotations

import pytest

from tests.plan_probe import Probe, abi, column
from vexq_b200 import plan as P


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
