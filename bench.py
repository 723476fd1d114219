#!/usr/bin/env python
"""Benchmark of the vexq hot path on B200: scan → filter → project →
aggregate over HBM-resident dictionary-coded columns.

Workload (one "step"): the 6,000,000-row lineitem-shaped table with
122,880-row row groups, two queries through the C ABI —
  (a) filtered GROUP BY flag,status with 8 aggregates   (44 B/row algorithmic)
  (b) five-range-predicate SUM(price*disc)               (28 B/row algorithmic)
Metric: GB/s scanned (algorithmic bytes = reference width of every
referenced column × rows in non-pruned row groups, ÷ device time).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl vexq|reference]

Under torchrun each rank owns its own 6M-row table (weak scaling, no
data-path collective); timing is the max over ranks.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

NROWS = 6_000_000
RG_ROWS = 122_880
WORKLOAD = "lineitem 6M rows (122,880-row row groups): Q1-shape GROUP BY + Q6-shape range SUM"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="vexq", choices=["vexq", "reference"])
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-extra", action="store_true", help="default line without the join and batch objects")
    ap.add_argument("--profile", nargs="?", const="lineitem", default=None,
                    choices=["lineitem", "groupby", "join", "radix", "batch", "filter"],
                    help="profiling driver, no timing: a short fixed launch sequence of one workload for ncu "
                         "(lineitem: 3 x Q1 and 3 x Q6 over 6M rows; groupby: dense and hash GROUP BY over 4M "
                         "rows; join: Q3/Q12 global-table joins; radix: the same partitioned; batch: 64 plans "
                         "batched; filter: selection bitmaps)")
    ap.add_argument("--workload", default="lineitem", choices=["lineitem", "batch", "serve"],
                    help="lineitem: Q1+Q6 step (default); batch: 256 Zipf GROUP BYs, batched vs one by one; "
                         "serve: Poisson arrivals of a Q1/Q6/Q3 mix over resident tables, p50/p99")
    ap.add_argument("--fact-rows", type=int, default=60_000_000, help="serve workload: fact and probe rows")
    ap.add_argument("--queries", type=int, default=400, help="serve workload: queries per arm")
    ap.add_argument("--plans", type=int, default=256, help="batch workload: number of GROUP BY plans")
    return ap.parse_args()


def serve_workload(args):
    """Serving: lineitem (fact) rows, orders (build) = fact/4 and items (probe)
    = fact rows resident in HBM; a 50/20/30 mix of the Q1-shape GROUP BY,
    the Q6-shape range SUM and the Q3-shape join with randomised date
    cutoffs, prepared once (64 plans); queries submitted to the serving loop.
    Arms: plain (one query per launch, one worker) and batched (continuous
    batching, two workers), closed loop (all queued at once: throughput) and
    open loop (Poisson arrivals at 70% of the plain arm's closed-loop rate:
    p50/p99 latency, submit to result ready)."""
    import ctypes as C
    import datetime

    import numpy as np

    from vexq_b200 import abi, build, datagen as D, exec as X, workloads as W
    build.build()
    X.init(0)
    fact = args.fact_rows
    h_li, h_o, h_it = D.lineitem(fact, seed=77, rg_rows=RG_ROWS), D.orders(fact // 4, seed=78), D.items(fact, fact // 4, seed=79)
    li, o, it = X.GpuTable(h_li), X.GpuTable(h_o), X.GpuTable(h_it)

    def day(n):
        return (datetime.date(1970, 1, 1) + datetime.timedelta(days=int(n))).isoformat()

    rng = np.random.default_rng(5)
    ops, kinds = [], []
    for _ in range(64):
        u = rng.random()
        if u < 0.5:
            ops.append(X.GpuHashAggregate(li, W.q1_plan(day(8036 + rng.integers(1500, 2526)))))
            kinds.append("q1")
        elif u < 0.7:
            lo = 8036 + int(rng.integers(0, 2000))
            ops.append(X.GpuHashAggregate(li, W.q6_plan(day(lo), day(lo + 365))))
            kinds.append("q6")
        else:
            ops.append(X.GpuParallelHashJoinAggregate(o, it, W.q3_plan(float(rng.uniform(0.3, 0.6)), float(rng.uniform(0.3, 0.6)))))
            kinds.append("q3")
    alone = {}
    for op, k in zip(ops, kinds):
        op.run().close()
        t0 = time.perf_counter()
        op.run().close()
        alone.setdefault(k, []).append((time.perf_counter() - t0) * 1e3)
    L = abi.load()

    def arm(arrivals, workers, flags):
        srv = C.c_void_p()
        abi.check(L.vexq_server_start(1 << 37, 16, workers, flags, C.byref(srv)))
        order = rng.integers(0, len(ops), len(arrivals))
        tickets = []
        start = time.perf_counter()
        for a, qi in zip(arrivals, order):
            now = time.perf_counter() - start
            if a > now:
                time.sleep(a - now)
            tk = C.c_int64()
            abi.check(L.vexq_server_submit(srv, ops[qi].h, C.byref(tk)))
            tickets.append(tk.value)
        lat = []
        for tk in tickets:
            h = C.c_void_p()
            abi.check(L.vexq_server_wait(srv, tk, 600000, C.byref(h)))
            L.vexq_result_free(h)
            ms = C.c_double()
            abi.check(L.vexq_server_latency(srv, tk, C.byref(ms)))
            lat.append(ms.value)
        total = time.perf_counter() - start
        la, q, mb, mc = C.c_int64(), C.c_int64(), C.c_int32(), C.c_int32()
        abi.check(L.vexq_server_stats(srv, C.byref(la), C.byref(q), C.byref(mb), C.byref(mc)))
        abi.check(L.vexq_server_stop(srv))
        lat = np.array(lat)
        return {"qps": round(len(arrivals) / total, 2), "p50_ms": round(float(np.percentile(lat, 50)), 3),
                "p99_ms": round(float(np.percentile(lat, 99)), 3), "launches": la.value, "max_batch": mb.value,
                "max_concurrent": mc.value}

    n = args.queries
    closed_plain = arm(np.zeros(n), 1, abi.SERVE_NO_BATCH)
    closed_batched = arm(np.zeros(n), 2, 0)
    qps = 0.7 * closed_plain["qps"]
    arrivals = np.cumsum(rng.exponential(1.0 / qps, n))
    poisson_plain = arm(arrivals, 1, abi.SERVE_NO_BATCH)
    poisson_batched = arm(arrivals, 2, 0)
    # host-CPU baseline: the C++ restatement of the reference's parallel path
    # (all host threads) on one query of each kind from the same mix, the
    # mix's queries/s from their times weighted 50/20/30
    cpu = None
    if not args.no_cpu:
        from oracle import refcpu as R
        workers = os.cpu_count() or 1
        tli, to, tit = R.RefTable(h_li), R.RefTable(h_o), R.RefTable(h_it)
        secs = {}
        for k, mk in (("q1", lambda: W.q1_plan(day(8036 + 2000))), ("q6", lambda: W.q6_plan(day(9036), day(9401))),
                      ("q3", lambda: W.q3_plan(0.45, 0.45))):
            t0 = time.perf_counter()
            if k == "q3":
                R.join_raw(to, tit, mk(), workers=workers)
            else:
                R.agg_raw(tli, mk(), workers=workers)
            secs[k] = time.perf_counter() - t0
        per_query = 0.5 * secs["q1"] + 0.2 * secs["q6"] + 0.3 * secs["q3"]
        cpu = {"value": round(1.0 / per_query, 3), "unit": "queries/s", "cores": workers, "cpu": cpu_model(), "kind": "port",
               "sample": "one query of each kind on the same tables (C++ restatement of ParallelHashAggregate / "
                         "ParallelHashJoinAggregate), queries/s of the 50/20/30 mix from their times",
               "seconds": {k: round(v, 3) for k, v in secs.items()}}
    line = {"metric": "queries/s", "value": closed_batched["qps"], "unit": "queries/s", "n_gpus": 1,
            "steps": n, "warmup": 1, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic (seeded lineitem / orders / items generators)",
            "config": {"workload": f"serving: {fact} fact rows, {fact // 4} build rows, {fact} probe rows; "
                                   "50% Q1 / 20% Q6 / 30% Q3 with randomised cutoffs"},
            "alone_ms_median": {k: round(float(statistics.median(v)), 3) for k, v in alone.items()},
            "closed_plain": closed_plain, "closed_batched": closed_batched,
            "poisson_qps": round(qps, 2), "poisson_plain": poisson_plain, "poisson_batched": poisson_batched,
            "cpu_baseline": cpu}
    print(json.dumps(line), flush=True)


def batch_plans(nplans):
    """The batching workload's plans: rows log-uniform over 10K-4M, key
    cardinality log-uniform over 2-65,536 with Zipf(1.1) frequencies as
    dictionary codes, float64 values U(0,1e5) at 2 decimals, mixed
    SUM/COUNT/MIN/MAX/AVG. Returns (host tables, plans)."""
    import math

    import numpy as np

    from vexq_b200 import datagen as D, plan as P
    rng = np.random.default_rng(2024)
    mixes = [lambda v: [P.sum_(v, "sum"), P.count_star("count")],
             lambda v: [P.min_(v, "min"), P.max_(v, "max"), P.count_star("count")],
             lambda v: [P.avg(v, "avg"), P.sum_(v, "sum")],
             lambda v: [P.sum_(v, "sum"), P.count_star("count"), P.min_(v, "min"), P.max_(v, "max"), P.avg(v, "avg")]]
    hosts, plans = [], []
    for i in range(nplans):
        rows = int(math.exp(rng.uniform(math.log(1e4), math.log(4e6))))
        card = int(round(math.exp(rng.uniform(math.log(2), math.log(65536)))))
        mix = int(rng.integers(4))
        hosts.append(D.zipf_groups(rows, card, seed=i))
        plans.append(P.AggPlan(None, [0], mixes[mix](P.col(1))))
    return hosts, plans


def batch_leg(nplans, steps, warmup, peak, cpu=True):
    """One step = every plan of the batching workload. The batched arm (one
    persistent launch per path class, graph replay, autotuned) against the
    same plans one by one through vexq_plan_run; device time is the kernels
    alone: the batch's graph between CUDA events on its stream, with the group
    tables' results written over PCIe and before the copy back of the rest; the
    plans one by one by the device clock inside their kernels. The CPU
    figure is one pass of the C++ restatement of ParallelHashAggregate over
    every plan on all host threads."""
    from vexq_b200 import exec as X
    hosts, plans = batch_plans(nplans)
    tabs = [X.GpuTable(h) for h in hosts]
    ops = [X.GpuHashAggregate(t, p) for t, p in zip(tabs, plans)]

    def plain():
        ms, nbytes = 0.0, 0
        for op in ops:
            r = op.run()
            ms += r.kernel_ms
            nbytes += r.bytes_scanned
            r.close()
        return ms, nbytes

    for _ in range(max(warmup, 3)):
        plain()
    pms = []
    for _ in range(steps):
        ms, nbytes = plain()
        pms.append(ms)
    b = X.GpuBatch(ops, autotune=True)
    for _ in range(max(warmup, 3)):
        for r in b.exec():
            r.close()
    bms, walls = [], []
    for _ in range(steps):
        t0 = time.perf_counter()
        res = b.exec()
        walls.append(time.perf_counter() - t0)
        for r in res:
            r.close()
        bms.append(b.stats()[1])
    explain = b.explain()
    b.close()
    for op in ops:
        op.close()
    p_ms, b_ms = statistics.median(pms), statistics.median(bms)
    out = {"workload": f"{nplans} GROUP BYs, 10K-4M rows, 2-65,536 groups, Zipf(1.1)",
           "bytes_per_step": nbytes, "rows_per_step": sum(h.nrows for h in hosts),
           "batched": {"value": round(nbytes / b_ms / 1e6, 3), "unit": "GB/s", "ms_per_step": round(b_ms, 4),
                       "frac_of_peak": round(nbytes / b_ms / 1e6 / peak, 4),
                       "wall_ms_per_step": round(statistics.median(walls) * 1e3, 3)},
           "plain_one_by_one": {"value": round(nbytes / p_ms / 1e6, 3), "unit": "GB/s", "ms_per_step": round(p_ms, 4)},
           "batched_over_plain": round(p_ms / b_ms, 3), "tuning": explain}
    if cpu:
        from oracle import refcpu as R
        workers = os.cpu_count() or 1
        rts = [R.RefTable(h) for h in hosts]
        t0 = time.perf_counter()
        for rt, pl in zip(rts, plans):
            R.agg_raw(rt, pl, workers=workers)
        cdt = time.perf_counter() - t0
        out["cpu_baseline"] = {"value": round(nbytes / cdt / 1e9, 3), "unit": "GB/s", "ms_per_step": round(cdt * 1e3, 1),
                               "cores": workers, "cpu": cpu_model(), "kind": "port",
                               "sample": "one pass over every plan (C++ restatement of ParallelHashAggregate)"}
    return out


def batch_workload(args):
    """256 independent GROUP BYs (batch_leg) as their own JSON line."""
    from vexq_b200 import build, exec as X
    build.build()
    X.init(0)
    peaks, _ = measured_peaks()
    leg = batch_leg(args.plans, args.steps, args.warmup, float(peaks.get("hbm_gbs", 6650.0)), cpu=not args.no_cpu)
    line = {"metric": "GB/s scanned", "value": leg["batched"]["value"], "unit": "GB/s", "n_gpus": 1,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": leg["batched"]["ms_per_step"],
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic (seeded Zipf(1.1) dictionary codes, 2-decimal values)",
            "config": {"workload": leg["workload"], "bytes_per_step": leg["bytes_per_step"], "batch": leg["tuning"]},
            **{k: leg[k] for k in ("batched", "plain_one_by_one", "batched_over_plain") if k in leg},
            "cpu_baseline": leg.get("cpu_baseline")}
    print(json.dumps(line), flush=True)


def join_leg(steps, warmup, peak, cpu=True):
    """The join workload on the plain drop-in: orders (1.5M rows, unique
    int64 keys) as the build side, items (6M rows, foreign keys uniform over
    the build keys) as the probe side, Q3 shape (GROUP BY key, SUM, top 10)
    and Q12 shape (mode IN list, date range, CASE counts by mode). Per query:
    device ms (CUDA events on the plan's stream around `steps` runs, host work
    between launches included) and the result's kernel ms; algorithmic bytes
    are the referenced columns of both sides. The CPU figure is the C++
    restatement of ParallelHashJoinAggregate on all host threads."""
    import torch

    from vexq_b200 import datagen as D, exec as X, workloads as W
    ho, hp = D.orders(1_500_000, seed=5), D.items(6_000_000, 1_500_000, seed=6)
    go, gp = X.GpuTable(ho), X.GpuTable(hp)
    stream = torch.cuda.Stream()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    out = {"workload": "orders 1.5M (build) x items 6M (probe), int64 keys"}
    rts = None
    if cpu:
        from oracle import refcpu as R
        rts = (R.RefTable(ho), R.RefTable(hp))
    for name, mk in (("q3", W.q3_plan), ("q12", W.q12_plan)):
        op = X.GpuParallelHashJoinAggregate(go, gp, mk())
        op.set_stream(stream.cuda_stream)
        for _ in range(max(warmup, 3)):
            op.run().close()
        torch.cuda.synchronize()
        kms, nbytes, launches = 0.0, 0, 0
        e0.record(stream)
        for _ in range(steps):
            r = op.run()
            kms += r.kernel_ms
            nbytes = r.bytes_scanned
            launches += r.launches
            r.close()
        e1.record(stream)
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / steps
        kms /= steps
        q = {"device_ms": round(ms, 4), "kernel_ms": round(kms, 4), "bytes": nbytes,
             "gbs": round(nbytes / ms / 1e6, 1), "kernel_gbs": round(nbytes / kms / 1e6, 1),
             "frac_of_peak": round(nbytes / kms / 1e6 / peak, 4), "launches_per_query": launches / steps,
             "plan": op.explain()}
        op.close()
        if rts is not None:
            from oracle import refcpu as R
            workers = os.cpu_count() or 1
            R.join_raw(rts[0], rts[1], mk(), workers=workers)
            reps, t0 = 0, time.perf_counter()
            while reps < 2 or (time.perf_counter() - t0 < 4.0 and reps < 10):
                R.join_raw(rts[0], rts[1], mk(), workers=workers)
                reps += 1
            cdt = (time.perf_counter() - t0) / reps
            q["cpu_port_ms"] = round(cdt * 1e3, 2)
            q["cpu_port_gbs"] = round(nbytes / cdt / 1e9, 3)
        out[name] = q
    if rts is not None:
        out["cpu_cores"] = os.cpu_count() or 1
    go.close()
    gp.close()
    return out


def profile_driver(kind="lineitem"):
    """Small fixed launch sequence for ncu (no timing): tables uploaded once,
    then a few runs of each plan of the chosen workload."""
    import numpy as np

    from vexq_b200 import build, datagen as D, exec as X, plan as P, workloads as W
    from vexq_b200.table import HostTable, float_column, int_column
    build.build()
    X.init(0)

    def runs(op, n):
        for _ in range(n):
            op.run().close()
        print(op.explain(), flush=True)
        op.close()

    if kind == "lineitem":
        gt = X.GpuTable(D.lineitem(NROWS, seed=43, rg_rows=RG_ROWS))
        for mk in (W.q1_plan, W.q6_plan):
            runs(X.GpuHashAggregate(gt, mk()), 3)
    elif kind == "groupby":
        # dense table over 65,536 and 1,000 Zipf(1.1) groups, then a hash table
        # over 200,000 distinct int64 keys (4M rows each)
        for card in (65536, 1000):
            runs(X.GpuHashAggregate(X.GpuTable(D.zipf_groups(4_000_000, card, seed=7)), W.batch_plan()), 3)
        rng = np.random.default_rng(3)
        keys = rng.integers(0, 1 << 40, 200_000)[rng.integers(0, 200_000, 4_000_000)]
        vals = np.rint(rng.uniform(0, 1e7, 4_000_000)) / 100.0
        ht = HostTable([int_column("k", keys), float_column("v", vals)], 4_000_000, 65536)
        runs(X.GpuHashAggregate(X.GpuTable(ht), W.batch_plan()), 3)
    elif kind in ("join", "radix"):
        go, gi = X.GpuTable(D.orders(1_500_000, seed=5)), X.GpuTable(D.items(6_000_000, 1_500_000, seed=6))
        bits = 8 if kind == "radix" else 0
        runs(X.GpuParallelHashJoinAggregate(go, gi, W.q3_plan(radix_bits=bits)), 2)
        runs(X.GpuParallelHashJoinAggregate(go, gi, W.q12_plan(radix_bits=bits)), 2)
    elif kind == "batch":
        rng = np.random.default_rng(2024)
        ops = []
        for i in range(64):
            rows = int(np.exp(rng.uniform(np.log(1e4), np.log(4e6))))
            card = int(round(np.exp(rng.uniform(np.log(2), np.log(65536)))))
            ops.append(X.GpuHashAggregate(X.GpuTable(D.zipf_groups(rows, card, seed=i)), W.batch_plan()))
        b = X.GpuBatch(ops)
        for _ in range(2):
            for r in b.exec():
                r.close()
        print(b.explain(), flush=True)
        b.close()
        for op in ops:
            op.close()
    elif kind == "filter":
        gt = X.GpuTable(D.lineitem(NROWS, seed=43, rg_rows=RG_ROWS))
        for pred in (W.q6_plan().predicate, W.q1_plan().predicate):
            f = X.GpuFilter(gt, pred)
            for _ in range(3):
                f.bitmap()


def cpu_model() -> str:
    try:
        with open("/proc/cpuinfo") as f:
            for ln in f:
                if ln.startswith("model name"):
                    return ln.split(":", 1)[1].strip()
    except OSError:
        pass
    import platform
    return platform.processor() or "unknown"


def parity_report(gpu_rows, ref, names):
    """Float cells of one query against the oracle's serial fold (the
    reference's row-order result) and its exact sum. A cell whose distance to
    the serial fold exceeds 1e-12 relative passes only when the GPU value is
    within 1e-13 of the exact sum and the serial fold's own error explains
    the gap; such cells are listed by name."""
    import math
    ref_rows = ref.rows()
    worst = {"gpu_vs_serial": 0.0, "gpu_vs_exact": 0.0, "serial_vs_exact": 0.0}
    via_exact, ok = [], len(gpu_rows) == len(ref_rows)
    for i, (g, r) in enumerate(zip(gpu_rows, ref_rows)):
        for j, (a, b) in enumerate(zip(g, r)):
            if not isinstance(a, float) or not isinstance(b, float) or math.isnan(a) or math.isnan(b):
                ok = ok and (a == b or (isinstance(a, float) and isinstance(b, float)))
                continue
            ex = ref.exact[j][i]
            sc = max(abs(b), 1e-300)
            d = abs(a - b) / sc
            worst["gpu_vs_serial"] = max(worst["gpu_vs_serial"], d)
            if not math.isnan(ex):
                se = max(abs(ex), 1e-300)
                eg, er = abs(a - ex) / se, abs(b - ex) / se
                worst["gpu_vs_exact"] = max(worst["gpu_vs_exact"], eg)
                worst["serial_vs_exact"] = max(worst["serial_vs_exact"], er)
                if d > 1e-12:
                    passed = eg <= 1e-13 and abs(a - b) / se <= er + 1e-13
                    ok = ok and passed
                    via_exact.append({"row": i, "col": names[j], "gpu_vs_serial": d, "gpu_vs_exact": eg,
                                      "serial_vs_exact": er})
            elif d > 1e-12:
                ok = False
    return {"rows": len(gpu_rows), "pass": ok, **{k: float(f"{v:.3g}") for k, v in worst.items()},
            "cells_passing_via_exact_arbiter": via_exact}


def measured_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return json.load(f), "measured"
    except Exception:
        return {"hbm_gbs": 6650.0}, "fallback"


def profile_traffic():
    """Per-launch DRAM bytes of the dominant kernel from the committed ncu summary."""
    try:
        with open(os.path.join(ROOT, "profiles", "traffic.json")) as f:
            return json.load(f)
    except Exception:
        return {}


class ClockSampler:
    """nvidia-smi clocks and throttle reasons during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.lines = []
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = float(f[2])
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx,
                "reasons": sorted(reasons), "samples": len(sm)}


def workload_config(world, step_bytes):
    """The `config` object of both arms' line (the same workload, keys and values)."""
    return {"workload": WORKLOAD, "rows_per_gpu": NROWS, "rg_rows": RG_ROWS,
            "bytes_per_step_per_gpu": step_bytes, "parallelism": f"replicas{world}",
            "l2": "inputs (264 MB / 168 MB per query) exceed the 126 MB L2; no flush"}


def dist_setup(args):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return world, rank, local


def cpu_reference_step(tbl, plans, workers):
    from oracle import refcpu as R
    for pl in plans:
        R.agg_raw(tbl, pl, workers=workers)


def run_reference(args, world, rank):
    """The reference's CPU path (C++ restatement of ParallelHashAggregate,
    one row group per morsel, all host threads), same workload and metric."""
    if rank != 0:
        return
    from oracle import refcpu as R
    from vexq_b200 import datagen as D, workloads as W
    host = D.lineitem(NROWS, seed=43, rg_rows=RG_ROWS)
    tbl = R.RefTable(host)
    q1, q6 = W.q1_plan(), W.q6_plan()
    workers = os.cpu_count() or 1
    step_bytes = 44 * NROWS + 28 * NROWS
    for _ in range(max(args.warmup, 3)):
        cpu_reference_step(tbl, [q1, q6], workers)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        cpu_reference_step(tbl, [q1, q6], workers)
    dt = (time.perf_counter() - t0) / args.steps
    value = step_bytes / dt / 1e9
    line = {
        "impl": "reference", "metric": "GB/s scanned", "value": round(value, 3), "unit": "GB/s",
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(dt * 1e3, 3),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic (seeded lineitem-shaped generator)",
        "config": workload_config(world, step_bytes),
        "cpu_baseline": {"value": round(value, 3), "unit": "GB/s", "cores": workers, "kind": "port",
                         "sample": f"full workload per step ({NROWS} rows, Q1+Q6), {args.steps} steps"},
        "e2e": {"value": round(value, 3), "unit": "GB/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def main():
    args = parse()
    world, rank, local = dist_setup(args)
    if args.profile:
        profile_driver(args.profile)
        return
    if args.impl == "reference":
        run_reference(args, world, rank)
        return
    if args.workload in ("batch", "serve"):
        if rank == 0:
            (batch_workload if args.workload == "batch" else serve_workload)(args)
        return
    import datetime

    import torch
    import torch.distributed as dist

    torch.cuda.set_device(local)
    if world > 1:
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120), device_id=torch.device("cuda", local))
    from vexq_b200 import build, datagen as D, exec as X, workloads as W

    build.build()
    X.init(local)
    host = D.lineitem(NROWS, seed=43 + rank, rg_rows=RG_ROWS)
    gt = X.GpuTable(host)
    q1 = X.GpuHashAggregate(gt, W.q1_plan())
    q6 = X.GpuHashAggregate(gt, W.q6_plan())
    stream = torch.cuda.Stream()
    q1.set_stream(stream.cuda_stream)
    q6.set_stream(stream.cuda_stream)

    # Every step submits one Q1 and one Q6 run (vexq_plan_submit: returns
    # once the launches are queued) and then reads both results of the step
    # before it, so the host prepares each run while the one ahead of it
    # executes and the GPU never waits for the host. Submitting a plan again
    # settles its previous result first (the Q6 submit waits for the last
    # Q6, with this step's Q1 already queued behind it). All K steps' kernels
    # finish inside the timed region; the last step's results are read after.
    pending = []

    def read(r1, r6):
        out = (r1.bytes_scanned, r6.bytes_scanned, r1.scan_ms, r6.scan_ms, r1.launches + r6.launches)
        assert r1.nrows > 0 and r6.nrows == 1
        r1.close()
        r6.close()
        return out

    def step():
        pending.append((q1.submit(), q6.submit()))
        return read(*pending.pop(0)) if len(pending) > 1 else None

    from vexq_b200.replicas import job_rate_gbs, max_over_ranks, run_timed

    clocks = ClockSampler(local)
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)

    def barrier():
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()

    def start():
        clocks.start()
        time.sleep(0.3)
        ev0.record(stream)

    def stop():
        ev1.record(stream)
        torch.cuda.synchronize()
        return ev0.elapsed_time(ev1)

    ms, stats = run_timed(step, args.steps, args.warmup, start, stop, barrier)
    # the first timed step read the last warm-up step's results
    stats = stats[1:] + [read(*r) for r in pending]
    pending.clear()
    clk = clocks.stop()
    step_bytes = stats[0][0] + stats[0][1]
    q1_bytes = stats[0][0]
    q1_scan = statistics.mean(s[2] for s in stats)
    q6_scan = statistics.mean(s[3] for s in stats)
    launches = sum(s[4] for s in stats)
    max_ms = max_over_ranks(ms, dist if world > 1 else None, device="cuda")
    ms_step = max_ms / args.steps
    value = job_rate_gbs(step_bytes, world, ms_step)

    # ---- end to end: host buffers, H2D inside the timed region ----
    e2e = None
    if not args.no_e2e:
        cudart = torch.cuda.cudart()
        regs = []
        for c in host.columns:
            for a in (c.values, c.validity):
                if a is not None and a.nbytes:
                    cudart.cudaHostRegister(a.ctypes.data, a.nbytes, 0)
                    regs.append(a)
        h2d = sum(a.nbytes for a in regs)
        for _ in range(2):
            r = q1.run_host(host)
            r.close()
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()
        t0 = time.perf_counter()
        e2e_launches = 0
        d2h = 0
        for _ in range(args.steps):
            r1 = q1.run_host(host)
            r6 = q6.submit()
            r1.collect()
            r6.collect()
            d2h = 8 * (r1.nrows * r1.ncols + r6.nrows * r6.ncols)
            e2e_launches += r1.launches + r6.launches
            r1.close()
            r6.close()
        torch.cuda.synchronize()
        dt = (time.perf_counter() - t0) / args.steps
        dt = max_over_ranks(dt, dist if world > 1 else None, device="cuda")
        for a in regs:
            cudart.cudaHostUnregister(a.ctypes.data)
        e2e = {"value": round(step_bytes * world / dt / 1e9, 3), "unit": "GB/s", "h2d_bytes_per_step": h2d,
               "d2h_bytes_per_step": d2h, "ms_per_step": round(dt * 1e3, 3)}

    # ---- CPU baseline: the oracle's ParallelHashAggregate on host cores ----
    cpu = parity = None
    if rank == 0 and not args.no_cpu:
        from oracle import refcpu as R
        tbl = R.RefTable(host)
        workers = os.cpu_count() or 1
        plans = [W.q1_plan(), W.q6_plan()]
        cpu_reference_step(tbl, plans, workers)
        reps, t0 = 0, time.perf_counter()
        while reps < 3 or (time.perf_counter() - t0 < 10.0 and reps < 50):
            cpu_reference_step(tbl, plans, workers)
            reps += 1
        cdt = (time.perf_counter() - t0) / reps
        cpu = {"value": round(step_bytes / cdt / 1e9, 3), "unit": "GB/s", "cores": workers, "cpu": cpu_model(),
               "kind": "port",
               "sample": f"{reps} full steps ({NROWS} rows, Q1+Q6) of the C++ restatement of "
                         "ParallelHashAggregate, one row group per morsel"}
        # the same oracle as the checker: the serial fold and exact sums of
        # both queries against one GPU run of each
        parity = {}
        for name, op, pl in (("q1", q1, plans[0]), ("q6", q6, plans[1])):
            r = op.run()
            rows = r.rows()
            names = r.names
            r.close()
            parity[name] = parity_report(rows, R.agg(tbl, pl, workers=0), names)

    peaks, src = measured_peaks()
    peak = float(peaks.get("hbm_gbs", 6650.0))
    achieved = q1_bytes / (q1_scan / 1e3) / 1e9
    tr = profile_traffic().get("q1_scan_dram_bytes_per_launch")
    roof = {"bound": "hbm", "achieved": round(achieved, 1), "peak": peak, "unit": "GB/s",
            "frac": round(achieved / peak, 4), "traffic": tr, "peak_source": f"{src} hbm_gbs",
            "kernel": ("vq_agg (Q1 scan-filter-project-aggregate, one launch: every block adds its partials as exact "
                       "fixed-point atomics into one of 8 accumulator copies and the last block to finish writes the "
                       "merged row into pinned host memory; first block's start to that write, device clock)"),
            "q6_kernel_gbs": round(stats[0][1] / (q6_scan / 1e3) / 1e9, 1)}
    if rank == 0:
        line = {
            "metric": "GB/s scanned", "value": round(value, 3), "unit": "GB/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms_step, 4),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic (seeded lineitem-shaped generator, no TPC-H rows)",
            "config": workload_config(world, step_bytes),
            "rows_per_s": round(2 * NROWS * world / (ms_step / 1e3), 1),
            "kernel_only_gbs": round(step_bytes / ((q1_scan + q6_scan) / 1e3) / 1e9, 1),
            "roofline": roof, "cpu_baseline": cpu, "e2e": e2e, "gpu_launches": launches, "clocks": clk,
            "parity": parity,
        }
        if world == 1 and not args.no_extra:
            line["join"] = join_leg(max(5, args.steps // 2), args.warmup, peak, cpu=not args.no_cpu)
            line["batch"] = batch_leg(args.plans, max(3, args.steps // 4), args.warmup, peak, cpu=not args.no_cpu)
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
