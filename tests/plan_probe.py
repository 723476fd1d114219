"""Plans compiled on a host without a GPU (plan_probe.cpp): the tests that look
at what a plan's kernels compile to, at sizes no test table has."""
from __future__ import annotations

import ctypes as C
import os
import subprocess

from vexq_b200 import abi, build
from vexq_b200 import plan as P

HERE = os.path.dirname(os.path.abspath(__file__))
PACKAGE = os.path.dirname(os.path.abspath(build.__file__))


class Column(C.Structure):
    _fields_ = [("type", C.c_int32), ("nullable", C.c_int32), ("has_range", C.c_int32), ("finite", C.c_int32),
                ("dict", C.c_int64), ("imin", C.c_int64), ("imax", C.c_int64), ("fmin", C.c_double), ("fmax", C.c_double)]


def column(type_, nullable=False, dict_=0, lo=0, hi=1000, finite=True) -> Column:
    """A column whose values lie in [lo, hi] (STRING: dict_ dictionary entries)."""
    return Column(type_, nullable, 1, finite, dict_, int(lo), int(hi), float(lo), float(hi))


class Probe:
    def __init__(self, tmp: str):
        build.build()
        so = os.path.join(tmp, "plan_probe.so")
        subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(PACKAGE, "csrc"),
                               "-I", os.path.join(PACKAGE, "..", "include"), "-I", os.path.join(build.CUDA, "include"),
                               os.path.join(HERE, "plan_probe.cpp"), "-o", so, "-L", PACKAGE, "-lvexqcuda",
                               "-Wl,-rpath," + PACKAGE])
        L = self.lib = C.CDLL(so)
        L.probe_table.restype = C.c_void_p
        L.probe_table.argtypes = [C.c_int, C.c_void_p, C.c_int64]
        L.probe_table_free.argtypes = [C.c_void_p]
        L.probe_agg.argtypes = [C.c_void_p, C.c_void_p, C.c_char_p, C.c_int]
        L.probe_filter_key.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_int, C.c_char_p, C.c_int]
        L.probe_out_pool.restype = C.c_int64
        L.probe_out_pool.argtypes = [C.c_int, C.c_int64, C.c_int64, C.c_void_p]
        L.probe_agg_wide.argtypes = [C.c_void_p, C.c_void_p, C.c_char_p, C.c_int]
        L.probe_widen.argtypes = [C.c_void_p]
        L.probe_join.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_char_p, C.c_int]
        self.tables = []

    def table(self, columns, nrows: int):
        t = self.lib.probe_table(len(columns), (Column * len(columns))(*columns), nrows)
        self.tables.append(t)
        return t

    def agg(self, table, plan) -> str:
        """The plan's float-sum windows and explain text, or "error …"."""
        out = C.create_string_buffer(8192)
        self.lib.probe_agg(table, C.byref(plan.desc), out, len(out))
        return out.value.decode(errors="replace")

    def agg_wide(self, table, plan) -> str:
        """agg, with the kernel for tables of 2^31 - 1 slots or more."""
        out = C.create_string_buffer(8192)
        self.lib.probe_agg_wide(table, C.byref(plan.desc), out, len(out))
        return out.value.decode(errors="replace")

    def widen(self, op) -> None:
        """Gives a prepared plan that kernel."""
        assert self.lib.probe_widen(op.h) == 0

    def join(self, build_table, probe_table, plan) -> str:
        out = C.create_string_buffer(8192)
        self.lib.probe_join(build_table, probe_table, C.byref(plan.desc), out, len(out))
        return out.value.decode(errors="replace")

    def filter_key(self, table, pred, lit_strs=None) -> bytes:
        """The key a Filter call's plan is kept under; lit_strs: {node: text}
        put into lit_str whatever the node's kind."""
        arena, nodes, nn, ch, nc, root = P.predicate_arrays(pred)
        for i, s in (lit_strs or {}).items():
            nodes[i].lit_str = s
        out = C.create_string_buffer(8192)
        n = self.lib.probe_filter_key(table, nodes, nn, ch, nc, root, out, len(out))
        assert n > 0, out.value
        return out.raw[:n]

    def out_pool(self, n: int, bytes_: int, lend_most: int):
        """(pinned bytes, blocks lent) of a result pool that gave n blocks out; needs a GPU."""
        lent = C.c_int32()
        return self.lib.probe_out_pool(n, bytes_, lend_most, C.byref(lent)), lent.value

    def close(self):
        for t in self.tables:
            self.lib.probe_table_free(t)


def lsb(text: str):
    return [int(x) for x in text.split("lsb=")[1].split()[0].split(",")]


__all__ = ["Probe", "column", "lsb", "abi"]
