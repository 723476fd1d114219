"""Timed cases of the library's query paths on one GPU.

A case is one prepared query (or one batch of them) over tables resident in
HBM, run the way a program that embeds the library runs it: the plan is made
once, each pass runs it and reads the result batch by batch through the C ABI's
views (vexq_result_next), as the cgo shim of a vexq build does. Sizes are those
of the benchmark's and the test suite's workloads (10K to 60M rows), odd ones
among them. Inputs are synthetic with the distributions of
vexq_b200/datagen.py, drawn on the GPU from the seed.
"""
from __future__ import annotations

import ctypes as C
import datetime
import math

import numpy as np
import torch

from vexq_b200 import abi, datagen as D, exec as X, plan as P, workloads as W
from vexq_b200.table import HostColumn, HostTable, date_column, float_column, int_column, pack_validity

ZIPF = 1.1


def listed():
    return [
        # a dashboard tile over a small table: launch and call latency
        {"name": "q1_10k", "kind": "q1", "rows": 10_000, "rg": 65_536, "cut": 0.966},
        # the benchmark's filtered GROUP BY with eight aggregates
        {"name": "q1_6m", "kind": "q1", "rows": 6_000_000, "rg": 122_880, "cut": 0.966},
        # the same over the serving workload's fact table
        {"name": "q1_60m", "kind": "q1", "rows": 60_000_000, "rg": 122_880, "cut": 0.966},
        # the benchmark's five-range-predicate sum (a selective global aggregate)
        {"name": "q6_6m", "kind": "q6", "rows": 6_000_000, "rg": 122_880, "cut": 0.3},
        # GROUP BY a dictionary-coded key, Zipf frequencies, all five aggregates
        {"name": "group_4m_1k", "kind": "group", "rows": 4_000_000, "rg": 65_536, "groups": 1_000, "mix": "all", "nulls": 0.0},
        # the same with NULLs in key and value, odd sizes, and a result of many batches
        {"name": "group_1m2_20k_null", "kind": "group", "rows": 1_234_567, "rg": 65_536, "groups": 20_011, "mix": "all", "nulls": 0.1},
        # top customers: GROUP BY a wide int64 key, ORDER BY the sum LIMIT 100
        {"name": "topk_4m_200k", "kind": "topk", "rows": 4_000_000, "rg": 65_536, "keys": 200_000, "limit": 100},
        # the benchmark's two joins: GROUP BY the join key with a top 10, and
        # CASE counts by mode
        {"name": "q3_6m", "kind": "q3", "build": 1_500_000, "rows": 6_000_000, "rg": 65_536, "cut": 0.48},
        {"name": "q12_6m", "kind": "q12", "build": 1_500_000, "rows": 6_000_000, "rg": 65_536},
        # a page of dashboard queries in one launch: many GROUP BYs over tables of their own
        {"name": "batch_32", "kind": "batch", "plans": 32, "rows": 2_000_000, "groups": 4_096, "rg": 65_536},
        # export of the rows a selective filter keeps, with computed columns
        {"name": "project_3m", "kind": "project", "rows": 3_000_001, "rg": 65_536, "cut": 0.3},
        # a selection bitmap for a host operator
        {"name": "filter_6m", "kind": "filter", "rows": 6_000_000, "rg": 122_880, "cut": 0.5},
    ]


def _log(rng, lo, hi):
    n = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    return n + rng.choice((0, 0, 1, 3, 6))


def draw(rng):
    kind = rng.choice(("q1", "q6", "group", "group", "topk", "q3", "q12", "batch", "project", "filter"))
    rg = rng.choice((65_536, 122_880))
    if kind == "q1":
        return {"kind": kind, "rows": _log(rng, 2_000, 16_000_000), "rg": rg, "cut": round(rng.uniform(0.3, 1.0), 3)}
    if kind in ("q6", "filter"):
        return {"kind": kind, "rows": _log(rng, 10_000, 16_000_000), "rg": rg, "cut": round(rng.uniform(0.05, 0.7), 3)}
    if kind == "group":
        n = _log(rng, 10_000, 4_000_000)
        return {"kind": kind, "rows": n, "rg": 65_536, "groups": min(_log(rng, 2, 65_536), n // 2),
                "mix": rng.choice(("sum_count", "min_max", "avg_sum", "all")), "nulls": rng.choice((0.0, 0.1))}
    if kind == "topk":
        return {"kind": kind, "rows": _log(rng, 100_000, 4_000_000), "rg": 65_536, "keys": _log(rng, 10_000, 500_000),
                "limit": rng.choice((10, 100, 1_000))}
    if kind in ("q3", "q12"):
        b = _log(rng, 10_000, 1_500_000)
        c = {"kind": kind, "build": b, "rows": int(b * rng.uniform(2.0, 4.0)), "rg": 65_536}
        return dict(c, cut=round(rng.uniform(0.3, 0.6), 3)) if kind == "q3" else c
    if kind == "batch":
        return {"kind": kind, "plans": rng.randrange(4, 33), "rows": _log(rng, 50_000, 2_000_000),
                "groups": _log(rng, 64, 16_384), "rg": 65_536}
    return {"kind": kind, "rows": _log(rng, 10_000, 4_000_000), "rg": rg, "cut": round(rng.uniform(0.05, 0.7), 3)}


# ---- inputs -----------------------------------------------------------------------


class _Rng:
    """Column generators on the GPU, handed out as numpy arrays."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))

    def ints(self, lo, hi, n):
        return torch.randint(lo, hi, (n,), generator=self.g, device="cuda")

    def uniform(self, n):
        return torch.rand(n, generator=self.g, device="cuda", dtype=torch.float64)

    def perm(self, n):
        return torch.randperm(n, generator=self.g, device="cuda")


def _np(x, dtype):
    return x.to(dtype).cpu().numpy()


def _dict(entries):
    b = [e.encode() for e in entries]
    off = np.zeros(len(b) + 1, dtype=np.uint32)
    np.cumsum([len(e) for e in b], out=off[1:])
    return off, np.frombuffer(b"".join(b), dtype=np.uint8).copy()


def _strings(name, idx, universe, rg):
    """A STRING column with a dictionary per row group, each in an order of its own (row group r starts at entry r)."""
    n, card = idx.numel(), len(universe)
    n_rg = -(-n // rg)
    r = torch.arange(n, device="cuda") // rg
    off, data = _dict([universe[(k + g) % card] for g in range(n_rg) for k in range(card)])
    return HostColumn(name, abi.TYPE_STRING, _np((idx - r) % card, torch.int32).view(np.uint32), None,
                      np.arange(n_rg + 1, dtype=np.uint32) * card, off, data)


def _lineitem(rows, rg, seed, same_keep=False):
    """same_keep: the filtered columns hold the same rows for every seed, in an order of the seed's own, so that a filter
    keeps equally many."""
    r = _Rng(seed)
    f = _Rng(rows) if same_keep else r
    flag, status = r.ints(0, 4, rows).clamp_(max=2), r.ints(0, 2, rows)
    qty = f.ints(1, 51, rows)
    disc = f.ints(0, 11, rows).double() / 100.0
    ship = f.ints(0, 2526, rows) + D.EPOCH_1992_01_02
    if same_keep:
        order = r.perm(rows)
        qty, disc, ship = qty[order], disc[order], ship[order]
    price = (qty * (900.0 + r.uniform(rows) * 104_100.0)).round_() / 100.0
    tax = r.ints(0, 9, rows).double() / 100.0
    return HostTable([_strings("l_returnflag", flag, D.FLAGS, rg), _strings("l_linestatus", status, D.STATUS, rg),
                      int_column("l_quantity", _np(qty, torch.int64)), float_column("l_extendedprice", _np(price, torch.float64)),
                      float_column("l_discount", _np(disc, torch.float64)), float_column("l_tax", _np(tax, torch.float64)),
                      date_column("l_shipdate", _np(ship, torch.int32))], rows, rg)


def _orders_items(build, rows, rg, seed):
    r = _Rng(seed)
    o = HostTable([int_column("o_orderkey", _np(r.perm(build) + 1, torch.int64)),
                   date_column("o_orderdate", _np(r.ints(0, D.DATE_SPAN, build) + D.EPOCH_1992_01_01, torch.int32)),
                   _strings("o_orderpriority", r.ints(0, 5, build), D.PRIORITIES, rg)], build, rg)
    qty = r.ints(1, 51, rows)
    price = (qty * (900.0 + r.uniform(rows) * 104_100.0)).round_() / 100.0
    it = HostTable([int_column("l_orderkey", _np(r.ints(1, build + 1, rows), torch.int64)),
                    date_column("l_shipdate", _np(r.ints(0, D.DATE_SPAN, rows) + D.EPOCH_1992_01_01, torch.int32)),
                    float_column("l_extendedprice", _np(price, torch.float64)),
                    float_column("l_discount", _np(r.ints(0, 11, rows).double() / 100.0, torch.float64)),
                    _strings("l_shipmode", r.ints(0, 7, rows), D.MODES, rg)], rows, rg)
    return o, it


def _zipf(rows, groups, rg, nulls, seed):
    r = _Rng(seed)
    p = torch.arange(1, groups + 1, device="cuda", dtype=torch.float64) ** -ZIPF
    cdf = torch.cumsum(p, 0)
    rank = torch.searchsorted(cdf / cdf[-1], r.uniform(rows), right=True).clamp_(max=groups - 1)
    code = r.perm(groups)[rank]
    once = r.perm(rows)[:groups]  # every group has a row
    code[once] = torch.arange(groups, device="cuda")
    # codes in first-occurrence order, as the writer gives them out
    first = torch.full((groups,), rows, device="cuda").scatter_reduce_(0, code, torch.arange(rows, device="cuda"), "amin")
    code = torch.argsort(torch.argsort(first))[code]
    val = (r.uniform(rows) * 1e7).round_() / 100.0
    vk = vv = None
    if nulls:
        vk = r.uniform(rows) >= nulls / 2
        vk[once] = True
        vk, vv = _np(vk, torch.bool), _np(r.uniform(rows) >= nulls, torch.bool)
    off, data = _dict(["k%05d" % i for i in range(groups)])
    codes = _np(code, torch.int32).view(np.uint32)
    if vk is not None:
        codes = np.where(vk, codes, np.uint32(0xFFFFFFFF))
    return HostTable([HostColumn("g_key", abi.TYPE_STRING, codes, pack_validity(vk), None, off, data),
                      float_column("g_value", _np(val, torch.float64), vv)], rows, rg)


def _wide_keys(rows, keys, rg, seed):
    r = _Rng(seed)
    pool = r.ints(0, 1 << 40, keys)
    val = (r.uniform(rows) * 1e7).round_() / 100.0
    return HostTable([int_column("c_key", _np(pool[r.ints(0, keys, rows)], torch.int64)),
                      float_column("c_value", _np(val, torch.float64))], rows, rg)


def _batch_sizes(case, k):
    """Rows and groups of plan k of a batch: spread over the logarithms of 10K..rows and 2..groups."""
    n = max(case["plans"] - 1, 1)
    rows = 10_000 * (case["rows"] / 10_000) ** (k / n)
    groups = 2 * (case["groups"] / 2) ** (((k * 7) % case["plans"]) / n)
    return int(rows), min(max(2, int(round(groups))), int(rows) // 2)


MIXES = ("sum_count", "min_max", "avg_sum", "all")


def _mix(mix):
    v = P.col(1)
    return {"sum_count": [P.sum_(v, "sum"), P.count_star("count")],
            "min_max": [P.min_(v, "min"), P.max_(v, "max"), P.count_star("count")],
            "avg_sum": [P.avg(v, "avg"), P.sum_(v, "sum")],
            "all": [P.sum_(v, "sum"), P.count_star("count"), P.min_(v, "min"), P.max_(v, "max"), P.avg(v, "avg")]}[mix]


def _day(frac):
    return int(D.EPOCH_1992_01_02 + round(frac * 2525))


def _iso(day):
    return (datetime.date(1970, 1, 1) + datetime.timedelta(days=day)).isoformat()


def _q6_days(case):
    lo = _day(case["cut"])
    return lo, lo + 365


def _q6_pred(case):
    lo, hi = _q6_days(case)
    return W.q6_plan(_iso(lo), _iso(hi)).predicate


def _tables(case, seed):
    """The host tables of a case."""
    k = case["kind"]
    if k in ("q1", "q6", "project", "filter"):
        return [_lineitem(case["rows"], case["rg"], seed, same_keep=k == "project")]
    if k == "group":
        return [_zipf(case["rows"], case["groups"], case["rg"], case["nulls"], seed)]
    if k == "topk":
        return [_wide_keys(case["rows"], case["keys"], case["rg"], seed)]
    if k in ("q3", "q12"):
        return list(_orders_items(case["build"], case["rows"], case["rg"], seed))
    return [_zipf(*_batch_sizes(case, i), case["rg"], 0.0, seed * 64 + i) for i in range(case["plans"])]


def prepare(case, seed):
    k = case["kind"]
    X.init(0)
    tabs = [X.GpuTable(h) for h in _tables(case, seed)]
    torch.cuda.empty_cache()
    if k == "q1":
        op = X.GpuHashAggregate(tabs[0], W.q1_plan(_iso(_day(case["cut"]))))
    elif k == "q6":
        lo, hi = _q6_days(case)
        op = X.GpuHashAggregate(tabs[0], W.q6_plan(_iso(lo), _iso(hi)))
    elif k == "group":
        op = X.GpuHashAggregate(tabs[0], P.AggPlan(None, [0], _mix(case["mix"])))
    elif k == "topk":
        op = X.GpuHashAggregate(tabs[0], P.AggPlan(None, [0], [P.sum_(P.col(1), "total"), P.count_star("n")],
                                                   order_col=1, descending=True, limit=case["limit"]))
    elif k == "q3":
        op = X.GpuParallelHashJoinAggregate(tabs[0], tabs[1], W.q3_plan(case["cut"], case["cut"] - 0.02))
    elif k == "q12":
        op = X.GpuParallelHashJoinAggregate(tabs[0], tabs[1], W.q12_plan())
    elif k == "batch":
        op = X.GpuBatch([X.GpuHashAggregate(t, P.AggPlan(None, [0], _mix(MIXES[i % 4]))) for i, t in enumerate(tabs)])
    elif k == "project":
        price, disc = P.col(D.L_PRICE), P.col(D.L_DISC)
        op = X.GpuProject(tabs[0], [P.col(D.L_SHIPDATE), P.col(D.L_QTY), price * (1 - disc), price * (1 - disc) * (1 + P.col(D.L_TAX))],
                          ["shipdate", "qty", "disc_price", "charge"], _q6_pred(case))
    else:
        op = X.GpuFilter(tabs[0], P.and_(P.col(D.L_SHIPDATE) <= P.lit(_iso(_day(case["cut"]))), P.between(P.col(D.L_DISC), 0.02, 0.08)))
    return {"kind": k, "op": op}


# ---- one pass -----------------------------------------------------------------------

_WIDTH = {abi.TYPE_INT64: 8, abi.TYPE_FLOAT64: 8, abi.TYPE_DATE: 4, abi.TYPE_STRING: 4, abi.TYPE_BOOL: 1}
_DTYPE = {abi.TYPE_INT64: np.int64, abi.TYPE_FLOAT64: np.float64, abi.TYPE_DATE: np.int32, abi.TYPE_STRING: np.int32, abi.TYPE_BOOL: np.uint8}


def _read(res):
    """Every batch of a result through the C ABI's views: per column its values, its validity bitmap's bytes and, for
    strings, the batches' dictionaries; copied out, since the views end with the next call."""
    lib, bv, at = abi.load(), abi.BatchView(), C.string_at
    nxt, ref, h = lib.vexq_result_next, C.byref(bv), res.h
    cols = None
    while True:
        abi.check(nxt(h, ref))
        n = bv.length
        if n == 0:
            break
        views = bv.cols
        if cols is None:
            cols = [(views[c].type, [], [], []) for c in range(bv.ncols)]
        nb = (n + 7) >> 3
        for c, (t, vals, valid, strs) in enumerate(cols):
            v = views[c]
            vals.append(at(v.values, n * _WIDTH[t]))
            valid.append(at(v.validity, nb))
            if t == abi.TYPE_STRING and v.dict_len:
                end = C.c_uint32.from_address(v.dict_str_off + 4 * v.dict_len).value
                strs.append(at(v.dict_bytes, end))
    res.close()
    out = []
    for t, vals, valid, strs in cols or []:
        o = [np.frombuffer(b"".join(vals), dtype=_DTYPE[t]), np.frombuffer(b"".join(valid), dtype=np.uint8)]
        if t == abi.TYPE_STRING:
            o.append(np.frombuffer(b"".join(strs), dtype=np.uint8))
        out.append(o)
    return out


def _flat(results):
    """The outputs of many results as one array a type."""
    f, i, b = [], [], []
    for cols in results:
        for c in cols:
            for a in c:
                (f if a.dtype == np.float64 else i if a.dtype != np.uint8 else b).append(a)
    return [np.concatenate(f), np.concatenate([a.astype(np.int64) for a in i]), np.concatenate(b)]


def run(state):
    k, op = state["kind"], state["op"]
    if k == "filter":
        bits, count = op.bitmap()
        return [np.frombuffer(bits, dtype=np.uint8), count]
    if k == "batch":
        return _flat([_read(r) for r in op.exec()])
    return _read(op.run())


# ---- what a pass cannot do without --------------------------------------------------


def work(case):
    k = case["kind"]
    n = case["rows"]
    if k == "q1":
        return {"bytes": 44 * n + 6 * 80, "flops": 11 * n}
    if k == "q6":
        return {"bytes": 28 * n + 8, "flops": 2 * n}
    if k == "group":
        return {"bytes": 12 * n + case["groups"] * 44, "flops": 4 * n}
    if k == "topk":
        return {"bytes": 16 * n + case["limit"] * 24, "flops": 2 * n}
    if k == "q3":
        return {"bytes": 12 * case["build"] + 28 * n + 160, "flops": 3 * n}
    if k == "q12":
        return {"bytes": 12 * case["build"] + 16 * n + 40, "flops": 2 * n}
    if k == "batch":
        s = [_batch_sizes(case, i) for i in range(case["plans"])]
        return {"bytes": sum(12 * r + 28 * g for r, g in s), "flops": sum(3 * r for r, _ in s)}
    if k == "project":
        return {"bytes": 36 * n + int(0.018 * n) * 28, "flops": 3 * n}
    return {"bytes": 12 * n + n // 8, "flops": 3 * n}


# ---- the same in 64 bits on the host ------------------------------------------------


def _col(t, i):
    return t.columns[i].values


def _codes(t, i):
    """Global dictionary index of every row of a _strings() column."""
    c = t.columns[i]
    card = int(c.dict_rg_first[1])
    return (c.values.astype(np.int64) + np.arange(t.nrows) // t.rg_rows) % card


def _groups(ids):
    """Rows sorted by group, each group's start, and the groups in output order: by first row, the NULL key (id -1) ahead
    of them."""
    order = np.argsort(ids, kind="stable")
    s = ids[order]
    starts = np.flatnonzero(np.r_[True, s[1:] != s[:-1]]) if len(s) else np.zeros(0, np.int64)
    return order, starts, np.argsort(np.where(s[starts] < 0, -1, order[starts]), kind="stable")


def _sums(v, order, starts, by):
    """Sums by group, summed in extended precision."""
    if not len(starts):
        return np.zeros(0)
    return np.add.reduceat(v.astype(np.longdouble)[order], starts)[by].astype(np.float64)


def _group_exact(t, mix):
    key, val = t.columns[0], t.columns[1]
    ids = key.values.view(np.int32).astype(np.int64)  # a NULL key is code -1
    ok = val.valid_mask(t.nrows)
    order, starts, by = _groups(ids)
    v = np.where(ok, val.values, 0.0)
    s = _sums(v, order, starts, by)
    nn = np.add.reduceat(ok.astype(np.int64)[order], starts)[by]
    mn = np.minimum.reduceat(np.where(ok, val.values, np.inf)[order], starts)[by]
    mx = np.maximum.reduceat(np.where(ok, val.values, -np.inf)[order], starts)[by]
    none = nn == 0
    avg = np.where(none, 0.0, s / np.maximum(nn, 1))
    mn, mx = np.where(none, 0.0, mn), np.where(none, 0.0, mx)
    return {"sum_count": [s, None], "min_max": [mn, mx, None], "avg_sum": [avg, s], "all": [s, None, mn, mx, avg]}[mix]


def exact(case, seed):
    k = case["kind"]
    if k in ("q12", "filter") or case["rows"] > 20_000_000:
        return None
    hosts = _tables(case, seed)
    t = hosts[0]
    none = [None, None]
    if k == "group":
        return [[None, None, None]] + [[a, None] for a in _group_exact(t, case["mix"])]
    if k == "batch":
        per = [_group_exact(h, MIXES[i % 4]) for i, h in enumerate(hosts)]
        return [np.concatenate([a for p in per for a in p if a is not None]), None, None]
    if k == "topk":
        order, starts, by = _groups(_col(t, 0))
        s = _sums(_col(t, 1), order, starts, by)
        return [none, [-np.sort(-s)[:case["limit"]], None], none]
    if k == "q3":
        o, it = hosts
        ok = np.zeros(case["build"] + 1, dtype=bool)
        ok[_col(o, 0)] = _col(o, 1) < D.join_mid(case["cut"])
        m = (_col(it, 1) > D.join_mid(case["cut"] - 0.02)) & ok[_col(it, 0)]
        order, starts, by = _groups(_col(it, 0)[m])
        s = _sums((_col(it, 2) * (1 - _col(it, 3)))[m], order, starts, by)
        return [none, [-np.sort(-s)[:10], None]]
    qty, price, disc, tax, ship = (_col(t, i) for i in (D.L_QTY, D.L_PRICE, D.L_DISC, D.L_TAX, D.L_SHIPDATE))
    if k == "q1":
        m = ship <= _day(case["cut"])
        qty, price, disc, tax = qty[m], price[m], disc[m], tax[m]
        g = _groups((_codes(t, D.L_FLAG) * 2 + _codes(t, D.L_STATUS))[m])
        cnt = np.diff(np.r_[g[1], len(qty)])[g[2]]
        dp = price * (1 - disc)
        sums = [_sums(v, *g) for v in (price, dp, dp * (1 + tax))]
        avgs = [_sums(v, *g) / cnt for v in (qty, price, disc)]
        return [[None] * 3, [None] * 3, none] + [[a, None] for a in sums + avgs] + [none]
    lo, hi = _q6_days(case)
    m = (ship >= lo) & (ship < hi) & (disc >= 0.05) & (disc <= 0.07) & (qty < 24)
    if k == "q6":
        return [[np.array([(price * disc)[m].astype(np.longdouble).sum()], dtype=np.float64), None]]
    dp = price[m] * (1 - disc[m])
    return [none, none, [dp, None], [dp * (1 + tax[m]), None]]
