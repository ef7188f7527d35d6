#!/usr/bin/env python
"""Benchmark of the B200 alignment stage (libsaruman_b200.so).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--config c2|c1|c4]

Metric: candidate alignments per second (every candidate pair aligned,
including those that score above k), with GCUPS (rectangle cells m*L per
second) beside it.  Default workload: the microbial-scale configuration --
5 Mbp seeded genome at 50 % GC with 40 repeat families of 1.5 kbp (5-50
copies, 99 % identity), 2M reads of 100 bp from both strands with 3 % errors
(70/15/15), k = 5; candidate windows are placed where the reference's q-gram
filter places them (read origin, plus the same offset in every other copy of
a repeat family), ~9.5 candidates per read as the reference's filter gives
on this genome.  Synthetic data: there is no network for real data.

One step aligns one such batch.  `value` times saru_align_device on inputs
already resident in HBM (one kernel launch per step; inputs ~4 GB, larger
than L2, so no flush is needed).  `e2e` times the same batch through the
public host entry point (saru_align_host) with pinned host buffers: host
validation, H2D of the inputs, the kernels, D2H of the scores and both
alignment-slot arrays, every step (the library overlaps the copies and the
kernels in slices of the call).

With torchrun (N > 1) each rank aligns its own batch (replicas, weak
scaling); rank 0 prints the max-over-ranks timing.  `--impl reference` times
the reference's own alignment code (src/cuda-functions.cu compiled for the
host, oracle/_ref) on all host cores over a bounded sample of the workload.
"""
from __future__ import annotations

import argparse
import dataclasses
import json
import os
import statistics
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

CONFIGS = {
    "c2": dict(workload="microbial-scale plain kernel: 5 Mbp repeat-rich genome, 2M reads x 100 bp, "
               "3% errors, k=5", genome=("repeat", 5_000_000, 201, "uniform"), reads=2_000_000,
               m=100, k=5, rate=0.03, mix=(0.70, 0.15, 0.15), unmapped=0.0),
    "c1": dict(workload="small: 1 Mbp uniform genome, 100k reads x 36 bp, 2% errors, k=2",
               genome=("uniform", 1_000_000, 101), reads=100_000, m=36, k=2, rate=0.02,
               mix=(0.70, 0.15, 0.15), unmapped=0.0),
    "c4": dict(workload="long-read-end stress: 10 Mbp uniform genome, 1M reads x 250 bp, 4% errors "
               "(60/20/20), 5% unmapped, k=15", genome=("uniform", 10_000_000, 401),
               reads=1_000_000, m=250, k=15, rate=0.04, mix=(0.60, 0.20, 0.20), unmapped=0.05),
    "c3": dict(workload="batching: 5 Mbp genome with Zipf(1.5, max 500) repeat copies (seed 313: "
               "1-112 copies per family), 4M reads of lengths {36,75,100,150} (1M each), 3% errors, "
               "k=ceil(0.06 m); every candidate the reference's filter makes (uneven count per "
               "read); all length bins in one batched request",
               genome=("repeat", 5_000_000, 313, "zipf"), reads=4_000_000, lengths=(36, 75, 100, 150),
               rate=0.03, mix=(0.70, 0.15, 0.15), unmapped=0.0),
    "c5": dict(workload="serving: 5 Mbp genome with Zipf(1.5, max 500) repeat copies (seed 313) "
               "resident on the device; Poisson arrivals of requests of 1k-500k reads (log-uniform), "
               "read lengths {36,75,100,150} in equal parts, k=ceil(0.06 m); requests carry reads "
               "only (the server filters, gathers and aligns); 60 GB device budget; continuous-"
               "batching server vs the plain per-request loop on one trace",
               genome=("repeat", 5_000_000, 313, "zipf"), reads=2_000_000,
               lengths=(36, 75, 100, 150), rate=0.03, mix=(0.70, 0.15, 0.15), unmapped=0.0,
               requests=400, min_reads=1_000, max_reads=500_000, budget=60 << 30, load=0.8),
}


def build_genome(cfg: dict):
    from saruman_b200 import workloads as W
    gs = cfg["genome"]
    if gs[0] == "uniform":
        return W.uniform_genome(gs[1], seed=gs[2]), None
    return W.repeat_genome_with_map(gs[1], seed=gs[2], copies=gs[3])


def build_batches(cfg: dict, rank: int, tables: list | None = None):
    """One batch per read-length bin (one for single-length configs) with
    candidates placed where the q-gram filter places them (synthetic, no
    GPU needed); the sequenced reads of each bin go to `tables` when given."""
    from saruman_b200 import workloads as W
    g, rmap = build_genome(cfg)
    lengths = cfg.get("lengths", (cfg.get("m"),))
    per_bin = cfg["reads"] // len(lengths)
    out = []
    for i, m in enumerate(lengths):
        k = cfg.get("k", W.k_for(m))
        rd = W.sample_reads(g, per_bin, m, cfg["rate"], seed=1000 + 17 * rank + i, mix=cfg["mix"],
                            unmapped=cfg["unmapped"])
        out.append(W.synthetic_candidates(g, rd, m, k, seed=2000 + 17 * rank + i, repeats=rmap,
                                          max_hits=cfg.get("max_hits", 1000)))
        if tables is not None:
            tables.append(rd.seqs)
    if tables is not None:
        tables.append(g)  # the genome last
    return out


def build_callsets(cfg: dict, rank: int, tables: list | None = None, info: dict | None = None):
    """One CallSet per read-length bin: the calls the reference's q-gram
    filter makes for the bin's reads on both strands (the library's device
    filter, which reproduces the reference's calls), at the reference's
    queue threshold for that read length.  Needs the library and a GPU (the
    filter runs on the calling thread's current device).  `info` receives
    the filter's device time and counts."""
    from saruman_b200 import workloads as W
    g, _ = build_genome(cfg)
    lengths = cfg.get("lengths", (cfg.get("m"),))
    per_bin = cfg["reads"] // len(lengths)
    out = []
    for i, m in enumerate(lengths):
        k = cfg.get("k", W.k_for(m))
        rd = W.sample_reads(g, per_bin, m, cfg["rate"], seed=1000 + 17 * rank + i, mix=cfg["mix"],
                            unmapped=cfg["unmapped"])
        cv = cfg.get("chunk_value") or W.chunk_value_for(m, k)
        cs = W.filter_callset(g, rd.seqs, m, k, cv)
        out.append(cs)
        if info is not None:
            info.setdefault("bins", []).append(
                {"m": m, "k": k, "reads": per_bin, "chunk_value": cv, "filter_ms": cs.filter_ms,
                 "candidates": cs.n, "calls": cs.ncalls, "perfect_hits": cs.perfect})
        if tables is not None:
            tables.append(rd.seqs)
    if tables is not None:
        tables.append(g)
    return out


def band_cells(b) -> int:
    """Cells of the band that must be evaluated per candidate: m*(2k+1)
    when only the end gap is free (so = 0), m*(4k+1) otherwise."""
    so_free = np.isin(b.dirs, (2, 3, 6, 7))
    per = np.where(so_free, b.m * (4 * b.k + 1), b.m * (2 * b.k + 1))
    return int(per.sum())


def rect_cells(b) -> int:
    return int((b.m * b.lengths).sum())


def algorithmic_bytes(b) -> int:
    """Bytes the stage must move per batch: read and window bytes, 9 bytes
    of offsets/flag per candidate in, 4-byte score and both alignment slots
    out."""
    return int(len(b.reads) + len(b.genome) + 9 * b.n + 4 * b.n + 2 * b.total_genome)


class ClockSampler:
    """nvidia-smi clocks and throttle reasons during the timed region."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                 "-lms", "200", "-i", str(self.device)], stdout=subprocess.PIPE,
                stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.proc = None
        time.sleep(0.3)
        return self

    def __exit__(self, *a):
        time.sleep(0.3)
        self.out = ""
        if self.proc:
            self.proc.terminate()
            try:
                self.out, _ = self.proc.communicate(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
                self.out = ""

    def summary(self) -> dict:
        sms, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in (self.out or "").splitlines():
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sms.append(float(f[1]))
                mx = float(f[2])
            except ValueError:
                continue
            for nm, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(nm)
        if not sms:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        return {"sm_mhz": statistics.median(sms), "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sms)}


def measured_peaks() -> dict:
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        return json.loads(p.read_text())
    return {"hbm_gbs": 6650.0, "fallback": True}


def profile_traffic() -> dict | None:
    """DRAM bytes per candidate of the diagonal kernel from the committed ncu
    summary (profiles/diag_kernel_c2.json), if present."""
    p = ROOT / "profiles" / "diag_kernel_c2.json"
    if p.exists():
        try:
            return json.loads(p.read_text())
        except ValueError:
            return None
    return None


def cpu_reference_rate(calls, seconds: float = 10.0, nthreads: int | None = None) -> dict:
    """The reference's own kernel code on the host (oracle/_ref), all host
    threads, over consecutive pieces of the workload's calls (each piece a
    call of its own, the layout the reference's host code would build for
    it) until `seconds`."""
    import ctypes as C
    lib_path = ROOT / "oracle" / "_ref" / "libref_emul.so"
    if not lib_path.exists():
        return {"value": None, "unavailable": "oracle/_ref/libref_emul.so not built"}
    lib = C.CDLL(str(lib_path))
    lib.ref_align_batch.restype = C.c_int
    nthreads = nthreads or os.cpu_count() or 1
    P = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    done = 0
    chunk = max(2000, 500 * nthreads)
    t0 = time.perf_counter()
    for b in calls:
        L = b.lengths
        gend = np.cumsum(L)
        for start in range(0, b.n, chunk):
            if time.perf_counter() - t0 >= seconds:
                break
            e = min(b.n, start + chunk)
            gs = int(gend[start - 1]) if start else 0
            Ls = L[start:e]
            go = np.cumsum(Ls).astype(np.int32)
            ro = ((np.arange(e - start) + 1) * b.m).astype(np.int32)
            esz = (b.m + 1) * (Ls + 1)
            eo = (np.cumsum(esz) - esz).astype(np.int32)
            gbytes = np.ascontiguousarray(b.genome[gs:int(gend[e - 1])])
            rbytes = np.ascontiguousarray(b.reads[start * b.m:e * b.m])
            dirs = np.ascontiguousarray(b.dirs[start:e])
            tot = int(go[-1]) + b.k * (e - start)
            sc = np.zeros(e - start, np.int32)
            ra = np.zeros(tot + 64, np.uint8)
            ga = np.zeros(tot + 64, np.uint8)
            rc = lib.ref_align_batch(C.c_int(0), C.c_int(1), P(gbytes), P(rbytes), P(go), P(ro),
                                     P(eo), C.c_int(e - start), P(dirs), C.c_int(b.k),
                                     C.c_size_t(tot), C.c_int(0), C.c_int(nthreads),
                                     C.c_int(256), P(sc), P(ra), P(ga))
            if rc != 0:
                return {"value": None, "unavailable": "reference host run failed"}
            done += e - start
        if time.perf_counter() - t0 >= seconds:
            break
    dt = time.perf_counter() - t0
    return {"value": done / dt, "cores": nthreads, "candidates": done, "seconds": dt}


def all_calls(css) -> list:
    return [cs.call(c) for cs in css for c in range(cs.ncalls)]


def run_reference_arm(args, cfg, rank: int) -> None:
    if rank != 0:
        return
    import torch
    torch.cuda.set_device(0)  # the workload's calls come from the device filter
    css = build_callsets(cfg, 0)
    calls = all_calls(css)
    per_step = []
    cores = None
    for i in range(args.warmup + args.steps):
        r = cpu_reference_rate(calls, seconds=args.ref_seconds)
        if r.get("value") is None:
            print(json.dumps({"impl": "reference", "unavailable": r.get("unavailable")}))
            return
        cores = r["cores"]
        if i >= args.warmup:
            per_step.append((r["candidates"], r["seconds"]))
    cand = sum(c for c, _ in per_step)
    secs = sum(t for _, t in per_step)
    value = cand / secs
    line = {
        "impl": "reference", "metric": "alignments/s", "value": value, "unit": "alignments/s",
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": 1000 * secs / len(per_step), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "int16", "data": "synthetic",
        "config": {"workload": cfg["workload"], "sample": "consecutive pieces of the workload's "
                   f"calls, {args.ref_seconds:.0f} s of host work per step"},
        "cpu_baseline": {"value": value, "unit": "alignments/s", "cores": cores,
                         "kind": "reference", "sample": f"{cand} candidates"},
        "e2e": {"value": value, "unit": "alignments/s", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))


class DeviceCalls:
    """A CallSet's inputs and outputs resident on the device, with one C-ABI
    call per reference call (pointers into the set's arrays), and pinned
    host copies of the inputs and outputs for the end-to-end legs."""

    def __init__(self, cs, dev, S, status):
        import torch
        T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        pin = lambda a: torch.from_numpy(np.ascontiguousarray(a)).pin_memory()  # noqa: E731
        self.cs, m = cs, cs.m
        self.g, self.r, self.go, self.ro, self.d = (T(cs.genome), T(cs.reads),
                                                    T(cs.genome_offsets), T(cs.read_offsets),
                                                    T(cs.dirs))
        self.scores = torch.zeros(cs.n, dtype=torch.int32, device=dev)
        self.ra = torch.zeros(cs.total_slots + 64, dtype=torch.uint8, device=dev)
        self.ga = torch.zeros(cs.total_slots + 64, dtype=torch.uint8, device=dev)
        self.h_in = [pin(cs.genome), pin(cs.reads), pin(cs.genome_offsets), pin(cs.read_offsets),
                     pin(cs.dirs)]
        self.h_out = [torch.empty(cs.n, dtype=torch.int32).pin_memory(),
                      torch.empty(cs.total_slots + 64, dtype=torch.uint8).pin_memory(),
                      torch.empty(cs.total_slots + 64, dtype=torch.uint8).pin_memory()]
        self.rb = S.compact_record_bytes(cs.m, cs.k)
        self.rec = torch.empty(max(cs.n, 1) * self.rb, dtype=torch.uint8, device=dev)
        self.h_rec = torch.empty(max(cs.n, 1) * self.rb, dtype=torch.uint8).pin_memory()
        self.sbs, self.srs, self.crs, self.spans = [], [], [], []
        cb, gb, sbase = cs.call_begin, cs.gbase, cs.sbase
        for c in range(cs.ncalls):
            a, b = int(cb[c]), int(cb[c + 1])
            g0, g1, s0, s1 = int(gb[c]), int(gb[c + 1]), int(sbase[c]), int(sbase[c + 1])
            self.sbs.append(S.SaruBatch(self.g.data_ptr() + g0, self.r.data_ptr() + a * m,
                                        self.go.data_ptr() + 4 * a, self.ro.data_ptr() + 4 * a,
                                        self.d.data_ptr() + a, b - a, cs.k, 0, 1, 1, m, g1 - g0,
                                        s1 - s0))
            self.srs.append(S.SaruResult(self.scores.data_ptr() + 4 * a, self.ra.data_ptr() + s0,
                                         self.ga.data_ptr() + s0, status.data_ptr()))
            self.crs.append(S.SaruResult(self.scores.data_ptr() + 4 * a,
                                         self.rec.data_ptr() + a * self.rb, None,
                                         status.data_ptr()))
            self.spans.append((a, b, g0, g1, s0, s1))

    def host_call(self, c: int):
        """Call c as a Batch over the pinned host inputs, and an AlignResult
        over the pinned host outputs."""
        import saruman_b200 as S
        from saruman_b200 import workloads as W
        cs, m = self.cs, self.cs.m
        a, b, g0, g1, s0, s1 = self.spans[c]
        hg, hr, hgo, hro, hd = (t.numpy() for t in self.h_in)
        bt = W.Batch(m=m, k=cs.k, genome=hg[g0:g1], reads=hr[a * m:b * m],
                     genome_offsets=hgo[a:b], read_offsets=hro[a:b],
                     edit_offsets=cs.edit_offsets[a:b], dirs=hd[a:b], ids=cs.ids[a:b],
                     pos=cs.pos[a:b])
        sc, ra, ga = (t.numpy() for t in self.h_out)
        return bt, S.AlignResult(sc[a:b], ra[s0:s1], ga[s0:s1])

    def copy_in(self, c0: int, c1: int):
        """Inputs of calls [c0, c1) (contiguous in every array), on the
        current stream."""
        a, g0, m = self.spans[c0][0], self.spans[c0][2], self.cs.m
        b, g1 = self.spans[c1 - 1][1], self.spans[c1 - 1][3]
        for d, h, lo, hi in ((self.g, self.h_in[0], g0, g1), (self.r, self.h_in[1], a * m, b * m),
                             (self.go, self.h_in[2], a, b), (self.ro, self.h_in[3], a, b),
                             (self.d, self.h_in[4], a, b)):
            d[lo:hi].copy_(h[lo:hi], non_blocking=True)

    def copy_out(self, c0: int, c1: int):
        a, s0 = self.spans[c0][0], self.spans[c0][4]
        b, s1 = self.spans[c1 - 1][1], self.spans[c1 - 1][5]
        for h, d, lo, hi in ((self.h_out[0], self.scores, a, b), (self.h_out[1], self.ra, s0, s1),
                             (self.h_out[2], self.ga, s0, s1)):
            h[lo:hi].copy_(d[lo:hi], non_blocking=True)

    def copy_out_compact(self, c0: int, c1: int):
        a, b = self.spans[c0][0], self.spans[c1 - 1][1]
        self.h_out[0][a:b].copy_(self.scores[a:b], non_blocking=True)
        self.h_rec[a * self.rb:b * self.rb].copy_(self.rec[a * self.rb:b * self.rb],
                                                  non_blocking=True)

    def bytes_in(self) -> int:
        return sum(int(h.numel() * h.element_size()) for h in self.h_in)

    def bytes_out(self) -> int:
        return 4 * self.cs.n + 2 * self.cs.total_slots


def call_groups(dcs: list, per_group: int) -> list:
    """Consecutive calls of each set in groups of up to `per_group`:
    (set index, first call, end call)."""
    out = []
    for i, d in enumerate(dcs):
        for c0 in range(0, d.cs.ncalls, per_group):
            out.append((i, c0, min(d.cs.ncalls, c0 + per_group)))
    return out


def legacy_names(n_ids: int):
    """The caller-owned read_names table of the reference's host program for
    read ids 0..n_ids-1 (names "read<id>"), as the library walks it: a list
    of struct read_name_hash (src/util.h:350-354: int read_number; char
    name[60]; UT_hash_handle hh) linked by the handle's third pointer."""
    import ctypes as C
    esz = 64 + 6 * 8 + 8
    buf = np.zeros(n_ids * esz, np.uint8)
    base = buf.ctypes.data
    rec = buf.reshape(n_ids, esz)
    rec[:, 0:4] = np.arange(n_ids, dtype=np.int32).view(np.uint8).reshape(n_ids, 4)
    names = np.char.add(b"read", np.arange(n_ids).astype("S12"))
    nb = np.frombuffer(names.astype("S60").tobytes(), np.uint8).reshape(n_ids, 60)
    rec[:, 4:64] = nb
    nxt = base + (np.arange(n_ids, dtype=np.uint64) + 1) * esz
    nxt[-1] = 0
    rec[:, 80:88] = nxt.view(np.uint8).reshape(n_ids, 8)
    return buf, C.c_void_p(base)


def timed(stream, fn, steps, world, dist, dev):
    import torch
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(steps):
        fn()
    e1.record(stream)
    e1.synchronize()
    ms = e0.elapsed_time(e1)
    if world > 1:
        t = torch.tensor([ms], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    return ms / steps


class ReadPool:
    """Reads of every length bin, as sequenced; a request takes a contiguous
    range of reads from each bin (reads only: the server filters them)."""

    def __init__(self, tables: list, ks: list):
        self.tables, self.ks = tables, ks

    def make(self, reads: int, rng) -> list:
        sets = []
        for t, k in zip(self.tables, self.ks):
            r = max(1, reads // len(self.tables))
            off = int(rng.integers(0, max(1, t.shape[0] - r)))
            sets.append((t[off:off + r], k, 0))
        return sets


def run_trace(S, genome, reqs: list, arrivals_s, pipeline: bool, budget: int,
              compact: bool = False, warm: list | None = None) -> dict:
    """Submits reads-only requests at their arrival times (seconds after the
    start; None = all at once) to a fresh server and returns per-request
    latency from arrival to results in host memory, the makespan, the
    candidates the filter made and the server's counters."""
    import threading
    srv = S.Server(pipeline=pipeline, max_requests_per_launch=64, max_inflight=2,
                   budget_bytes=budget)
    try:
        srv.set_genome(genome)
        for sets in warm or []:  # builds each bin's q-gram index; not timed
            t = srv.submit_reads(sets, compact=compact)
            rc, _ = srv.wait(t, 3_600_000)
            if rc != S.SARU_OK:
                raise RuntimeError(S.last_error())
            srv.release(t)
        g0, l0 = srv.counters()
        tickets = [None] * len(reqs)
        err = []
        lock = threading.Condition()
        t0 = time.monotonic_ns() // 1000

        def submitter():
            try:
                for q, sets in enumerate(reqs):
                    if arrivals_s is not None:
                        delay = t0 / 1e6 + arrivals_s[q] - time.monotonic()
                        if delay > 0:
                            time.sleep(delay)
                    t = srv.submit_reads(sets, compact=compact)
                    with lock:
                        tickets[q] = t
                        lock.notify_all()
            except Exception as ex:  # surfaced below
                with lock:
                    err.append(ex)
                    lock.notify_all()

        th = threading.Thread(target=submitter)
        th.start()
        done_us, cand = [0] * len(reqs), 0
        for q in range(len(reqs)):
            with lock:
                while tickets[q] is None and not err:
                    lock.wait()
                if err:
                    break
                t = tickets[q]
            rc, st = srv.wait(t, 3_600_000)
            if rc != S.SARU_OK:
                raise RuntimeError(f"request {q}: {rc} {S.last_error()}")
            done_us[q] = st.done_us
            cand += srv.candidates(t)
            srv.release(t)
        th.join()
        if err:
            raise err[0]
        groups, launches = srv.counters()
    finally:
        srv.close()
    arr_us = [t0 + (int(a * 1e6) if arrivals_s is not None else 0) for a in
              (arrivals_s if arrivals_s is not None else [0] * len(reqs))]
    lat_ms = [(d - a) / 1000 for d, a in zip(done_us, arr_us)]
    return {"lat_ms": lat_ms, "makespan_s": (max(done_us) - t0) / 1e6, "candidates": cand,
            "groups": groups - g0, "launches": launches - l0}


def serving(S, cfg: dict, nreq: int, seed: int = 4242, compact_too: bool = False,
            clk=None) -> dict:
    """The serving workload: one seeded Poisson trace of reads-only requests
    through the continuous-batching server and the plain per-request loop,
    at `load` of the plain loop's capacity, and both at saturation."""
    from saruman_b200 import workloads as W
    g, _ = build_genome(cfg)
    lengths = cfg["lengths"]
    per_bin = cfg["reads"] // len(lengths)
    tables = [W.sample_reads(g, per_bin, m, cfg["rate"], seed=1000 + i, mix=cfg["mix"],
                             unmapped=cfg["unmapped"]).seqs for i, m in enumerate(lengths)]
    pool = ReadPool(tables, [W.k_for(m) for m in lengths])
    rng = np.random.default_rng(seed)
    sizes = np.exp(rng.uniform(np.log(cfg["min_reads"]), np.log(cfg["max_reads"]), nreq))
    sizes = sizes.astype(np.int64)
    reqs = [pool.make(int(x), rng) for x in sizes]
    warm = [pool.make(20_000, rng) for _ in range(3)]
    # the capacity probe draws its requests from the trace's own size
    # distribution (a fixed request size misjudges the plain loop's capacity
    # for the trace's mix of small and large requests)
    prng = np.random.default_rng(seed + 1)
    psizes = np.exp(prng.uniform(np.log(cfg["min_reads"]), np.log(cfg["max_reads"]),
                                 max(16, nreq // 4))).astype(np.int64)
    probe = [pool.make(int(x), prng) for x in psizes]
    budget = cfg["budget"]
    import torch
    free, _ = torch.cuda.mem_get_info()
    budget = int(min(budget, free - (8 << 30)))
    # the plain loop's capacity in reads/s, closed loop; measured on the
    # second pass: the first server trace of a process measured up to 3x
    # slower than the same trace run again, which understated capacity
    run_trace(S, g, probe, None, False, budget, warm=warm)
    cap = run_trace(S, g, probe, None, False, budget, warm=warm)
    plain_reads_s = sum(t.shape[0] for sets in probe for t, _, _ in sets) / cap["makespan_s"]
    lam = cfg["load"] * plain_reads_s / float(sizes.mean())
    gaps = rng.exponential(1.0 / lam, nreq)
    arrivals = np.cumsum(gaps) - gaps[0]
    if clk is not None:
        clk.__enter__()
    try:
        b = run_trace(S, g, reqs, arrivals, True, budget, warm=warm)
    finally:
        if clk is not None:
            clk.__exit__(None, None, None)
    p = run_trace(S, g, reqs, arrivals, False, budget, warm=warm)
    sb = run_trace(S, g, reqs, None, True, budget, warm=warm)
    sp = run_trace(S, g, reqs, None, False, budget, warm=warm)

    def pct(v, q):
        return float(np.percentile(np.asarray(v), q))

    n_cand = b["candidates"]
    out = {
        "requests": nreq, "reads": int(sizes.sum()), "candidates": n_cand,
        "offered_load": {"requests_per_s": lam, "reads_per_s": lam * float(sizes.mean()),
                         "fraction_of_plain_capacity": cfg["load"]},
        "latency_ms": {"p50": pct(b["lat_ms"], 50), "p99": pct(b["lat_ms"], 99),
                       "max": max(b["lat_ms"]), "throughput": n_cand / b["makespan_s"],
                       "groups": b["groups"], "launches": b["launches"]},
        "plain_latency_ms": {"p50": pct(p["lat_ms"], 50), "p99": pct(p["lat_ms"], 99),
                             "max": max(p["lat_ms"]), "throughput": n_cand / p["makespan_s"],
                             "launches": p["launches"]},
        "saturation": {"value": n_cand / sb["makespan_s"], "plain_value": n_cand / sp["makespan_s"],
                       "batched_over_plain": sp["makespan_s"] / sb["makespan_s"],
                       "makespan_s": sb["makespan_s"]},
        "p99_plain_over_batched": pct(p["lat_ms"], 99) / pct(b["lat_ms"], 99),
        "budget_bytes": budget,
        "what": "requests of reads only: the server runs the reference's q-gram filter on both "
                "strands, gathers windows from the resident genome, aligns and returns slot "
                "strings; latency from arrival to results in host memory; plain = one request "
                "at a time, filter, one launch per call, no overlap",
    }
    if compact_too:
        sbc = run_trace(S, g, reqs, None, True, budget, compact=True, warm=warm)
        spc = run_trace(S, g, reqs, None, False, budget, compact=True, warm=warm)
        out["compact"] = {"value": n_cand / sbc["makespan_s"],
                          "plain_value": n_cand / spc["makespan_s"],
                          "batched_over_plain": spc["makespan_s"] / sbc["makespan_s"]}
    return out


def run_serving(args, cfg, rank: int) -> None:
    import torch
    import saruman_b200 as S
    torch.cuda.set_device(0)
    S.load()
    nreq = args.requests or cfg["requests"]
    clk = ClockSampler(0)
    r = serving(S, cfg, nreq, compact_too=True, clk=clk)
    line = {
        "metric": "alignments/s", "value": r["saturation"]["value"], "unit": "alignments/s",
        "n_gpus": 1, "steps": 1, "warmup": 3, "ms_per_step": 1000 * r["saturation"]["makespan_s"],
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u8/int32",
        "data": "synthetic",
        "config": {"workload": cfg["workload"], "requests": nreq, "reads": r["reads"],
                   "candidates": r["candidates"], "device_budget_bytes": r["budget_bytes"],
                   "step": "the whole trace, submitted at once (saturation)",
                   "l2": "inputs > L2"},
        "e2e": {"value": r["saturation"]["value"], "unit": "alignments/s",
                "h2d_bytes_per_step": r["reads"], "d2h_bytes_per_step": None},
        "serving": r,
        "batched_over_plain": r["saturation"]["batched_over_plain"],
        "clocks": clk.summary(),
    }
    print(json.dumps(line))


def tune_callsets(dcs: list, status, sample_calls: int = 6) -> dict:
    """Autotunes the launch shape of every (read length, k) bin on the bin's
    largest call: the cost model (trained on the GPU from the committed
    B200 sweep) ranks the shapes, the tuner times its top 6 and the
    default, and installs the fastest."""
    from saruman_b200 import autotune as A
    from saruman_b200 import costmodel as CM
    t0 = time.perf_counter()
    model = CM.trained_on_sweep()
    t_train = time.perf_counter() - t0
    out = {}
    for d in dcs:
        cs = d.cs
        c = int(np.argmax(np.diff(cs.call_begin)))
        smp = A.Sample.wrap(cs.call(c), d.sbs[c], d.srs[c], status)
        r = A.tune_bin(smp, model=model, top=6)
        out[f"{cs.m},{cs.k}"] = {"shape": list(r["best"]), "trials": len(r["ms"]),
                                 "ms_sample": r["ms"][r["best"]],
                                 "default_ms_sample": r["default_ms"],
                                 "sample_candidates": int(cs.call_begin[c + 1] - cs.call_begin[c])}
    out["cost_model_train_s"] = t_train
    out["tune_s"] = time.perf_counter() - t0
    return out


def measure_calls(S, css: list, args, dev, world: int, dist, tune: bool = True,
                  legacy_steps: int = 0, clk_device: int | None = None) -> dict:
    """Times one workload of calls (CallSets, all resident): the batched
    request (every call in one saru_align_multi_device request, replayed from
    a CUDA graph), the plain per-call kernel (one launch per call), the
    batched end-to-end path (pinned host buffers, groups of calls overlapped
    on three streams), the plain end-to-end path (a thread per strand,
    saru_align_host per call) and, if asked, the drop-in entry."""
    import threading

    import torch
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    dcs = [DeviceCalls(cs, dev, S, status) for cs in css]
    n_cand = sum(cs.n for cs in css)
    sbs = [sb for d in dcs for sb in d.sbs]
    srs = [sr for d in dcs for sr in d.srs]
    ncalls = len(sbs)
    stream = torch.cuda.Stream(device=dev)
    sptr = stream.cuda_stream
    # launch shapes first: the scratch sizes depend on them
    if args.shape:
        shape = tuple(int(x) for x in args.shape.split(","))
        for cs in css:
            S.set_tuning(cs.m, cs.k, *shape)
        tuning = {f"{cs.m},{cs.k}": {"shape": list(shape), "trials": 0} for cs in css}
    else:
        tuning = tune_callsets(dcs, status) if tune else {}
    status.zero_()
    reqs = [(sbs[q:q + 192], srs[q:q + 192]) for q in range(0, ncalls, 192)]
    nscr = max(S.multi_scratch_bytes(rb) for rb, _ in reqs)
    scratch = torch.empty(nscr, dtype=torch.uint8, device=dev)

    def step_batched():  # every call of the step in one request (one launch per length class)
        for rb, rr in reqs:
            S.align_multi_device(rb, rr, status.data_ptr(), scratch.data_ptr(), nscr, sptr)

    nplain = max(S.scratch_bytes(sb.n, sb.max_read_length, sb.k) for sb in sbs)
    scratch_plain = torch.empty(nplain, dtype=torch.uint8, device=dev)

    def step_plain():  # one launch per call, in call order
        for sb, sr in zip(sbs, srs):
            S.align_device(sb, sr, scratch_plain.data_ptr(), nplain, sptr)

    with torch.cuda.stream(stream):
        for _ in range(args.warmup):
            step_batched()
    stream.synchronize()
    if int(status.item()) != 0:
        raise SystemExit(f"kernel status {int(status.item())}")
    graph = torch.cuda.CUDAGraph()
    launches0 = S.kernel_launches()
    with torch.cuda.graph(graph, stream=stream):
        step_batched()
    per_step_launches = S.kernel_launches() - launches0

    def step_graph():
        with torch.cuda.stream(stream):
            graph.replay()

    step_graph()
    stream.synchronize()
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    clk = ClockSampler(clk_device) if clk_device is not None else None
    if clk:
        clk.__enter__()
    try:
        ms_step = timed(stream, step_graph, args.steps, world, dist, dev)
    finally:
        if clk:
            clk.__exit__(None, None, None)
    torch.cuda.synchronize()
    if int(status.item()) != 0:
        raise SystemExit(f"kernel status {int(status.item())}")

    for _ in range(2):
        step_plain()
    stream.synchronize()
    ms_plain = timed(stream, step_plain, args.steps, world, dist, dev)

    # end to end, batched
    e2e_steps = args.e2e_steps or max(1, min(args.steps, 5))
    s_in, s_run, s_out = (torch.cuda.Stream(device=dev) for _ in range(3))
    groups = call_groups(dcs, args.calls_per_group)
    gscr = max(S.multi_scratch_bytes(dcs[i].sbs[c0:c1]) for i, c0, c1 in groups)
    scratch_g = torch.empty(gscr, dtype=torch.uint8, device=dev)

    def e2e_batched():
        for i, c0, c1 in groups:
            d = dcs[i]
            with torch.cuda.stream(s_in):
                d.copy_in(c0, c1)
            s_run.wait_stream(s_in)
            S.align_multi_device(d.sbs[c0:c1], d.srs[c0:c1], status.data_ptr(),
                                 scratch_g.data_ptr(), gscr, s_run.cuda_stream)
            s_out.wait_stream(s_run)
            with torch.cuda.stream(s_out):
                d.copy_out(c0, c1)

    def timed_streams(fn, steps):
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(s_in)
        for _ in range(steps):
            fn()
        s_out.wait_stream(s_in)
        s_out.wait_stream(s_run)
        e1.record(s_out)
        e1.synchronize()
        ms = e0.elapsed_time(e1)
        if world > 1:
            t = torch.tensor([ms], device=dev)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ms = float(t.item())
        return ms / steps

    e2e_batched()
    torch.cuda.synchronize()
    e_ms = timed_streams(e2e_batched, e2e_steps)
    if int(status.item()) != 0:
        raise SystemExit(f"kernel status {int(status.item())} (e2e)")

    # compact records instead of slot strings: the batched request on the
    # device (graph replay), and end to end with the records copied out
    crs = [cr for d in dcs for cr in d.crs]
    creqs = [(sbs[q:q + 192], crs[q:q + 192]) for q in range(0, ncalls, 192)]

    def step_compact():
        for rb_, rr in creqs:
            S.align_multi_device_compact(rb_, rr, status.data_ptr(), scratch.data_ptr(), nscr,
                                         sptr)

    with torch.cuda.stream(stream):
        step_compact()
    stream.synchronize()
    cgraph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(cgraph, stream=stream):
        step_compact()

    def step_cgraph():
        with torch.cuda.stream(stream):
            cgraph.replay()

    step_cgraph()
    stream.synchronize()
    ms_compact = timed(stream, step_cgraph, args.steps, world, dist, dev)

    def e2e_compact():
        for i, c0, c1 in groups:
            d = dcs[i]
            with torch.cuda.stream(s_in):
                d.copy_in(c0, c1)
            s_run.wait_stream(s_in)
            S.align_multi_device_compact(d.sbs[c0:c1], d.crs[c0:c1], status.data_ptr(),
                                         scratch_g.data_ptr(), gscr, s_run.cuda_stream)
            s_out.wait_stream(s_run)
            with torch.cuda.stream(s_out):
                d.copy_out_compact(c0, c1)

    e2e_compact()
    torch.cuda.synchronize()
    ec_ms = timed_streams(e2e_compact, e2e_steps)
    if int(status.item()) != 0:
        raise SystemExit(f"kernel status {int(status.item())} (compact)")
    del cgraph

    # end to end, plain: the reference's structure -- a thread per strand,
    # each submitting its calls one at a time through saru_align_host
    strands = {}
    for i, d in enumerate(dcs):
        for c in range(d.cs.ncalls):
            strands.setdefault(int(d.cs.strand[c]), []).append((i, c))
    views = {(i, c): dcs[i].host_call(c) for i, d in enumerate(dcs) for c in range(d.cs.ncalls)}

    def plain_strand(lane, items, err):
        try:
            for key in items:
                b, out = views[key]
                S.align_host(b, lane=lane, out=out)
        except Exception as ex:  # surfaced after the join
            err.append(ex)

    def e2e_plain():
        err = []
        th = [threading.Thread(target=plain_strand, args=(0 if st == 0 else 1, items, err))
              for st, items in strands.items()]
        for t in th:
            t.start()
        for t in th:
            t.join()
        if err:
            raise err[0]

    e2e_plain()
    torch.cuda.synchronize()
    t_p = time.perf_counter()
    for _ in range(e2e_steps):
        e2e_plain()
    torch.cuda.synchronize()
    p_ms = (time.perf_counter() - t_p) * 1e3 / e2e_steps
    if world > 1:
        t = torch.tensor([p_ms], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        p_ms = float(t.item())

    legacy = None
    if legacy_steps > 0:
        # lines the reference prints: one per candidate with score <= k
        expect = sum(int((d.h_out[0].numpy() <= d.cs.k).sum()) for d in dcs)
        legacy = legacy_leg(S, css, strands, legacy_steps, world, dist, dev)
        if legacy["lines_per_step"] != expect:
            raise SystemExit(f"drop-in entry printed {legacy['lines_per_step']} lines, "
                             f"expected {expect}")
    out = dict(n_cand=n_cand, ncalls=ncalls, ms_step=ms_step, per_step_launches=per_step_launches,
               ms_plain=ms_plain, e_ms=e_ms, p_ms=p_ms, e2e_steps=e2e_steps, legacy=legacy,
               ms_compact=ms_compact, ec_ms=ec_ms,
               d2h_compact=sum(4 * d.cs.n + d.cs.n * d.rb for d in dcs),
               tuning=tuning, groups=len(groups), clocks=clk.summary() if clk else None,
               h2d=sum(d.bytes_in() for d in dcs), d2h=sum(d.bytes_out() for d in dcs))
    del graph
    return out


def batched_plain(r: dict, world: int) -> dict:
    """The batched-vs-plain part of a line from measure_calls' result."""
    n = r["n_cand"]
    return {
        "plain": {
            "kernel": {"value": world * n / (r["ms_plain"] * 1e-3), "ms_per_step": r["ms_plain"],
                       "launches_per_step": r["ncalls"],
                       "what": "one saru_align_device launch per reference call, in call order"},
            "e2e": {"value": world * n / (r["p_ms"] * 1e-3), "ms_per_step": r["p_ms"],
                    "what": "the reference's structure: a thread per strand, each submitting its "
                            "calls one at a time through saru_align_host (synchronous copies "
                            "in, kernel, copies out), pinned host buffers, host clock"}},
        "batched_over_plain": {"kernel": r["ms_plain"] / r["ms_step"], "e2e": r["p_ms"] / r["e_ms"]},
    }


def run_aligner(args, cfg: dict, rank: int, world: int, local: int) -> None:
    import torch
    import torch.distributed as dist
    import saruman_b200 as S

    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        from datetime import timedelta
        dist.init_process_group("nccl", timeout=timedelta(seconds=300), device_id=dev)
    S.load()
    winfo = {}
    t_build = time.perf_counter()
    css = build_callsets(cfg, rank, info=winfo)
    t_build = time.perf_counter() - t_build
    int_peak = S.int32_issue_peak() if rank == 0 else None
    r = measure_calls(S, css, args, dev, world, dist, tune=not args.no_tune,
                      legacy_steps=args.legacy_steps, clk_device=local)
    n_cand, ms_step = r["n_cand"], r["ms_step"]
    launches = r["per_step_launches"] * args.steps
    value = world * n_cand / (ms_step * 1e-3)
    e2e_value = world * n_cand / (r["e_ms"] * 1e-3)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()
    if rank != 0:
        return

    # ---- mixed read lengths (a reduced C3) and serving (a reduced C5) -------
    mixed = serve = None
    if world == 1 and args.config == "c2" and args.mixed_reads > 0:
        mcfg = dict(CONFIGS["c3"], reads=args.mixed_reads)
        mcss = build_callsets(mcfg, 0)
        mr = measure_calls(S, mcss, args, dev, 1, dist, tune=not args.no_tune)
        mixed = {"workload": CONFIGS["c3"]["workload"] + f" (reduced to {args.mixed_reads} reads)",
                 "candidates_per_step": mr["n_cand"], "calls_per_step": mr["ncalls"],
                 "read_lengths": [cs.m for cs in mcss], "k": [cs.k for cs in mcss],
                 "value": mr["n_cand"] / (mr["ms_step"] * 1e-3), "ms_per_step": mr["ms_step"],
                 "launches_per_step": mr["per_step_launches"],
                 "e2e": {"value": mr["n_cand"] / (mr["e_ms"] * 1e-3), "ms_per_step": mr["e_ms"]},
                 "tuning": mr["tuning"]}
        mixed.update(batched_plain(mr, 1))
        del mcss
    if world == 1 and args.config == "c2" and args.serve_requests > 0:
        serve = serving(S, CONFIGS["c5"], args.serve_requests)
        serve["workload"] = CONFIGS["c5"]["workload"] + \
            f" (reduced to {args.serve_requests} requests)"

    # ---- roofline --------------------------------------------------------
    peaks = measured_peaks()
    cells = sum(band_cells(cs) for cs in css)
    achieved_ops = 6 * cells / (ms_step * 1e-3)
    abytes = sum(algorithmic_bytes(cs) for cs in css)
    prof = profile_traffic() if args.config == "c2" else None
    traffic = None
    if prof and prof.get("dram_bytes_per_candidate"):
        traffic = prof["dram_bytes_per_candidate"] * n_cand
    roofline = {
        "bound": "int32",
        "achieved": achieved_ops / 1e12,
        "peak": int_peak / 1e12 if int_peak and int_peak > 0 else None,
        "unit": "Tops/s", "frac": (achieved_ops / int_peak) if int_peak and int_peak > 0 else None,
        "traffic": traffic,
        "traffic_source": "profiles/diag_kernel_c2.json (ncu dram bytes per candidate, small case, "
                          "scaled by candidates)" if traffic else None,
        "peak_source": "measured live by saru_int32_issue_probe on this GPU",
        "ops_per_candidate_definition": "band cells x 6 (m*(2k+1) or m*(4k+1) cells)",
        "hbm": {"achieved_gbs": abytes / (ms_step * 1e-3) / 1e9,
                "peak_gbs": peaks.get("hbm_gbs"),
                "frac": abytes / (ms_step * 1e-3) / 1e9 / peaks["hbm_gbs"],
                "algorithmic_bytes_per_step": abytes,
                "peak_source": "MEASURED_PEAKS.json" if not peaks.get("fallback") else "fallback"},
    }
    cpu = None
    if world == 1:
        cr = cpu_reference_rate(all_calls(css), seconds=args.cpu_seconds)
        if cr.get("value") is None:
            cpu = {"value": None, "unavailable": cr.get("unavailable")}
        else:
            cpu = {"value": cr["value"], "unit": "alignments/s", "cores": cr["cores"],
                   "kind": "reference",
                   "sample": f"{cr['candidates']} candidates: consecutive pieces of the "
                             "workload's calls, the reference's own kernel code compiled for "
                             f"the host, {args.cpu_seconds:.0f} s"}
    bins = winfo.get("bins", [])
    filt_ms = sum(b["filter_ms"] for b in bins)
    filt_reads = sum(2 * b["reads"] for b in bins)
    line = {
        "metric": "alignments/s", "value": value, "unit": "alignments/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_step,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u8/int32",
        "data": "synthetic",
        "config": {"workload": cfg["workload"], "candidates_per_step": n_cand,
                   "calls_per_step": r["ncalls"], "reads_per_step": cfg["reads"],
                   "read_lengths": [cs.m for cs in css], "k": [cs.k for cs in css],
                   "candidates": "the reference's q-gram filter on all reads, both strands "
                                 "(the library's device filter); calls cut at the reference's "
                                 "queue threshold", "bins": bins,
                   "parallelism": f"replicas x{world}", "l2": "inputs 4+ GB > L2, no flush",
                   "tuning": r["tuning"] or "default shapes", "build_s": t_build},
        "gcups_rect": world * sum(rect_cells(cs) for cs in css) / (ms_step * 1e-3) / 1e9,
        "gpu_launches": int(launches),
        "launch": "one CUDA graph replay per step "
                  f"({r['per_step_launches']} kernel launch(es) captured for {r['ncalls']} calls)",
        "e2e": {"value": e2e_value, "unit": "alignments/s", "h2d_bytes_per_step": r["h2d"],
                "d2h_bytes_per_step": r["d2h"], "steps": r["e2e_steps"],
                "what": f"pinned host buffers; {r['groups']} groups of up to "
                        f"{args.calls_per_group} calls, each copied in, aligned in one batched "
                        "request (saru_align_multi_device) and copied out, overlapped on three "
                        "streams; CUDA events"},
        "roofline": roofline,
        "cpu_baseline": cpu,
        "filter": {"value": filt_reads / (filt_ms * 1e-3) if filt_ms else None,
                   "unit": "read-strands/s", "reads": filt_reads // 2, "strands": 2,
                   "ms": filt_ms, "candidates": n_cand,
                   "what": "saru_filter_run on every read of the step, both strands: device "
                           "time incl. read upload, copy-back and call assembly"},
        "clocks": r["clocks"],
    }
    line.update(batched_plain(r, world))
    line["compact"] = {
        "value": world * n_cand / (r["ms_compact"] * 1e-3), "ms_per_step": r["ms_compact"],
        "roofline_frac": (6 * cells / (r["ms_compact"] * 1e-3) / int_peak
                          if int_peak and int_peak > 0 else None),
        "e2e": {"value": world * n_cand / (r["ec_ms"] * 1e-3), "unit": "alignments/s",
                "h2d_bytes_per_step": r["h2d"], "d2h_bytes_per_step": r["d2h_compact"]},
        "what": "saru_align_multi_device_compact: 2-bit traceback records per candidate instead "
                "of the slot strings (saru_expand_compact rebuilds the slots on the host); "
                "end to end as e2e, records copied out"}
    if r["legacy"]:
        line["e2e_legacy"] = r["legacy"]
    if mixed:
        line["mixed_lengths"] = mixed
    if serve:
        line["serving"] = serve
    print(json.dumps(line))


def legacy_leg(S, css, strands: dict, steps: int, world: int, dist, dev) -> dict:
    """cuda_needleman_wunsch per call, as src/hash.c:1094-1108 calls it:
    from one thread per strand, pageable host arrays, results printed by the
    library's writer before the call returns (stdout to /dev/null here)."""
    import ctypes as C
    import threading
    lib = S.load()
    n_ids = max(int(cs.ids.max()) + 1 for cs in css if cs.n)
    names, head = legacy_names(n_ids)
    C.c_void_p.in_dll(lib, "read_names").value = head.value
    C.c_ushort.in_dll(lib, "read_length_value").value = max(cs.m for cs in css)
    ctl = [(C.c_char * n_ids)(), (C.c_char * n_ids)()]
    C.c_void_p.in_dll(lib, "forward_output_control").value = C.addressof(ctl[0])
    C.c_void_p.in_dll(lib, "reverse_output_control").value = C.addressof(ctl[1])
    P = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    calls = {}
    for st in strands:
        calls[st] = []
        for cs in css:
            for c in range(cs.ncalls):
                if int(cs.strand[c]) == st:
                    calls[st].append(cs.call(c))
    n_cand = sum(b.n for v in calls.values() for b in v)

    def strand(st, bl):
        for b in bl:
            lib.cuda_needleman_wunsch(C.c_int(0), C.c_int(1), P(b.genome), P(b.reads),
                                      P(b.genome_offsets), P(b.read_offsets),
                                      P(b.edit_offsets), C.c_int(b.n), P(b.ids), P(b.pos),
                                      P(b.dirs), C.c_int(b.k), C.c_size_t(b.total_genome),
                                      C.c_size_t(b.n * b.m), C.c_size_t(b.total_edit),
                                      C.c_int(st))

    def one():
        th = [threading.Thread(target=strand, args=(st, bl)) for st, bl in calls.items()]
        for t in th:
            t.start()
        for t in th:
            t.join()

    libc = C.CDLL(None)
    sys.stdout.flush()
    libc.fflush(None)
    saved_out, saved_err = os.dup(1), os.dup(2)
    null = os.open(os.devnull, os.O_WRONLY)
    os.dup2(null, 1)
    os.dup2(null, 2)  # the per-call banner the reference prints on stderr
    try:
        for name in ("forward_alignments_done", "reverse_alignments_done"):
            C.c_uint.in_dll(lib, name).value = 0
        one()
        libc.fflush(None)
        printed = sum(C.c_uint.in_dll(lib, nm).value for nm in
                      ("forward_alignments_done", "reverse_alignments_done"))
        t0 = time.perf_counter()
        for _ in range(steps):
            one()
        libc.fflush(None)
        ms = (time.perf_counter() - t0) * 1e3 / steps
    finally:
        os.dup2(saved_out, 1)
        os.dup2(saved_err, 2)
        os.close(null)
        os.close(saved_out)
        os.close(saved_err)
    C.c_void_p.in_dll(lib, "read_names").value = None
    del names
    if world > 1:
        import torch
        t = torch.tensor([ms], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    return {"value": world * n_cand / (ms * 1e-3), "unit": "alignments/s", "ms_per_step": ms,
            "steps": steps, "lines_per_step": int(printed),
            "what": "cuda_needleman_wunsch per reference call from a thread per strand, "
                    "pageable host arrays, TSV lines written to /dev/null before each call "
                    "returns; host clock"}


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=("ours", "reference"), default="ours")
    ap.add_argument("--config", choices=sorted(CONFIGS), default="c2")
    ap.add_argument("--e2e-steps", type=int, default=None)
    ap.add_argument("--legacy-steps", type=int, default=2,
                    help="steps of the drop-in entry leg (0: skip)")
    ap.add_argument("--calls-per-group", type=int, default=12,
                    help="calls per group of the batched end-to-end leg")
    ap.add_argument("--mixed-reads", type=int, default=1_000_000,
                    help="reads of the mixed-length leg of the default line (0: skip)")
    ap.add_argument("--serve-requests", type=int, default=100,
                    help="requests of the serving leg of the default line (0: skip)")
    ap.add_argument("--cpu-seconds", type=float, default=10.0)
    ap.add_argument("--ref-seconds", type=float, default=10.0)
    ap.add_argument("--no-tune", action="store_true",
                    help="keep the default launch shapes (no autotuning)")
    ap.add_argument("--shape", default=None,
                    help="W,C,B: install this launch shape for every bin instead of tuning")
    ap.add_argument("--requests", type=int, default=None,
                    help="requests in the serving trace (c5)")
    ap.add_argument("--reads", type=int, default=None,
                    help="override the reads per step (smaller cases for profiling)")
    args = ap.parse_args()
    cfg = dict(CONFIGS[args.config])
    if args.reads:
        cfg["reads"] = args.reads
        cfg["workload"] += f" (reduced to {args.reads} reads)"

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference_arm(args, cfg, rank)
        return
    if args.config == "c5":
        if world > 1:
            raise SystemExit("the serving workload runs on one GPU")
        run_serving(args, cfg, rank)
        return
    run_aligner(args, cfg, rank, world, local)


if __name__ == "__main__":
    main()
