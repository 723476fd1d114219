"""GPU tests of GpuFilter.bitmap over ranges that end past the table (a caller
that walks a table in fixed steps): the table's bits, then zeros to the length
asked for; every byte against the oracle. A table loaded from a .vxq file has no
host copy whose length could tell."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import refcpu as R
from oracle import vxq_writer as VW
from tests.test_gpu_select import nullable_table
from vexq_b200 import plan as P

pytestmark = pytest.mark.gpu


def dirty(n):
    # freed blocks of the result's size hold ones: memory handed out next is not clear by luck
    blocks = [bytes(bytearray(b"\xff") * max(1, (n + 7) // 8)) for _ in range(64)]
    del blocks


@pytest.mark.parametrize("rows,lo,hi", [(100, 0, 8_900), (100, 0, 101), (100, 3, 8_903), (100, 99, 5_000), (100, 100, 164),
                                        (30_011, 16_384, 32_768), (30_011, 30_003, 30_100), (30_011, 29_998, 400_000), (30_011, 0, 30_011)])
@pytest.mark.parametrize("loaded", [False, True])
def test_bits_past_the_table_are_zero(gpu_lib, tmp_path, rows, lo, hi, loaded):
    X = gpu_lib
    host = nullable_table(n=rows)
    if loaded:
        path = str(tmp_path / "t.vxq")
        VW.write_vxq(path, host)
        t = X.GpuTable.from_vxq(path)
    else:
        t = X.GpuTable(host)
    for pred in (P.col(0) > 10, P.col(0) > -1_000_000):
        bits = np.unpackbits(np.frombuffer(R.filter_bits(R.RefTable(host), pred)[0], dtype=np.uint8), bitorder="little")[lo:rows]
        rows_asked = np.zeros(hi - lo, np.uint8)
        rows_asked[:len(bits)] = bits
        want = np.packbits(rows_asked, bitorder="little").tobytes()
        f = X.GpuFilter(t, pred)
        for _ in range(3):
            dirty(hi - lo)
            got, cnt = f.bitmap(lo, hi)
            assert cnt == int(bits.sum())
            assert len(got) == (hi - lo + 7) // 8
            assert got == want
    t.close()
