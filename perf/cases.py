"""The work that users of the library have it do, as timed cases.

A case is one pass through a public entry point: one alignment call on the
device (`device`), a batched request of calls of several read lengths
(`multi`, slot strings or compact records), a call from and to host memory
(`host`), the q-gram filter of a read batch on both strands (`filter`), or a
request of reads to the server (`server`).  Reads are sampled from seeded
genomes (uniform, or with repeat families) with sequencing errors; the
candidates of the alignment cases are the ones the q-gram filter makes for
them, so about 40 % of them score above k, as in real runs.

All outputs are whole numbers and bytes.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import saruman_b200 as S
from saruman_b200 import workloads as W

# candidates the filter makes per read (both strands), for sizes and bytes
PER_READ = {"uniform": 0.55, "repeat": 9.3}


def listed() -> list[dict]:
    return [
        # the smallest calls: a filter flush that holds a few reads
        dict(name="call_36_tiny", kind="device", m=36, k=2, n=54, genome="uniform", glen=1_000_000,
             rate=0.02, odd=0.0),
        # a whole small run: 100k reads of 36 bp on a 1 Mbp genome
        dict(name="call_36", kind="device", m=36, k=2, n=54_628, genome="uniform", glen=1_000_000,
             rate=0.02, odd=0.0),
        # one call at the filter's queue threshold for 100 bp reads
        dict(name="call_100", kind="device", m=100, k=5, n=176_000, genome="repeat",
             glen=5_000_000, rate=0.03, odd=0.0),
        # an odd read length and count, a band of more than 32 diagonals, Ns in some reads
        dict(name="call_133_n", kind="device", m=133, k=8, n=40_961, genome="repeat",
             glen=5_000_000, rate=0.03, codes="N", odd=0.003),
        # long read ends: one call of 250 bp at k = 15
        dict(name="call_250", kind="device", m=250, k=15, n=28_000, genome="repeat",
             glen=10_000_000, rate=0.04, odd=0.0),
        # a batched request of uneven calls of all read lengths
        dict(name="request_mixed", kind="multi", lengths="36,75,100,150", k=0, n=100_000,
             genome="repeat", glen=5_000_000, rate=0.03, compact=False),
        # a large batched request: 100k reads of 100 bp
        dict(name="request_100", kind="multi", lengths="100", k=5, n=930_000, genome="repeat",
             glen=5_000_000, rate=0.03, compact=False),
        # the same with compact records, the wire format of results
        dict(name="request_100_compact", kind="multi", lengths="100", k=5, n=930_000,
             genome="repeat", glen=5_000_000, rate=0.03, compact=True),
        # a call from and to host memory, as the reference's host program makes it
        dict(name="host_100", kind="host", m=100, k=5, n=176_000, genome="repeat",
             glen=5_000_000, rate=0.03, odd=0.0),
        # a host call some of whose reads hold several IUPAC codes: the exact path
        dict(name="host_36_iupac", kind="host", m=36, k=2, n=20_000, genome="uniform",
             glen=1_000_000, rate=0.02, codes="NRYK", odd=0.01),
        # candidate generation for a read batch, both strands
        dict(name="filter_100", kind="filter", m=100, k=5, reads=200_000, genome="repeat",
             glen=5_000_000, rate=0.03),
        # a serving request of reads of all lengths: filter, gather, align, results
        dict(name="server_reads", kind="server", lengths="36,75,100,150", k=0, reads=16_000,
             genome="repeat", glen=5_000_000, rate=0.03, compact=False),
    ]


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["device", "device", "device", "multi", "host", "filter", "server"])
    genome = rng.choice(["uniform", "repeat"])
    glen = _log(rng, 800_000, 5_000_000)
    rate = round(rng.uniform(0.01, 0.04), 4)
    if kind in ("multi", "server"):
        lengths = sorted({_log(rng, 36, 160) for _ in range(rng.choice([1, 2, 4]))})
        case = dict(kind=kind, lengths=",".join(map(str, lengths)), k=0, genome=genome, glen=glen,
                    rate=rate, compact=rng.random() < 0.5)
        if kind == "multi":
            case["n"] = _log(rng, 300, 200_000)
        else:
            case["reads"] = _log(rng, 1_000, 12_000)
        return case
    m = _log(rng, 36, 400)
    k = min(15, max(1, math.ceil(m * rng.uniform(0.03, 0.06))))
    case = dict(kind=kind, m=m, k=k, genome=genome, glen=glen, rate=rate)
    if kind == "filter":
        case["reads"] = _log(rng, 1_000, 100_000)
        return case
    case["n"] = _log(rng, 33, min(500_000, 3e8 / (m * k)))
    case["odd"] = 0.0
    if rng.random() < 0.3:
        case["odd"] = round(rng.uniform(0.001, 0.004), 4)
        case["codes"] = rng.choice(["N", "N", "NRYK"])
    if kind == "host":
        # reads with several IUPAC codes send a host call to the exact path,
        # whose matrices one call holds whole
        case["n"] = min(case["n"], 150_000_000 // ((m + 1) * (m + 2 * k + 1)))
    return case


# ---------------------------------------------------------------------------


class Kept:
    """What a program keeps between calls; a handle is given back with it."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        if "filter" in self.__dict__:
            S.load().saru_filter_destroy(self.filter)
        if "server" in self.__dict__:
            S.load().saru_server_destroy(self.server)


def _most(case: dict, reads: int) -> int:
    """Candidates a program leaves room for, one strand's or one set's."""
    return int((2 + 2 * PER_READ[case["genome"]]) * reads) + 50_000


def _genome(case: dict, seed: int) -> np.ndarray:
    if case["genome"] == "uniform":
        return W.uniform_genome(case["glen"], seed)
    return W.repeat_genome(case["glen"], seed, families=max(2, case["glen"] // 125_000))


def _reads(case: dict, genome: np.ndarray, m: int, n: int, seed: int) -> np.ndarray:
    """Reads as sequenced; a base is one of the IUPAC `codes` at rate `odd`."""
    seqs = W.sample_reads(genome, n, m, case["rate"], seed).seqs
    odd = case.get("odd", 0.0)
    if odd > 0:
        rng = np.random.default_rng(seed)
        at = rng.random(seqs.shape) < odd
        codes = np.frombuffer(case["codes"].encode(), np.uint8)
        seqs[at] = codes[rng.integers(0, len(codes), int(at.sum()))]
    return seqs


def _candidates(case: dict, genome: np.ndarray, m: int, k: int, n: int, seed: int):
    """The first n candidates the filter makes for sampled reads:
    (reads, read index, position, flag)."""
    reads, ids, pos, dirs, have = [], [], [], [], 0
    base, part = 0, int(1.1 * n / PER_READ[case["genome"]]) + 64
    # windows longer than the genome's tail are not made; an IUPAC code in a
    # read costs it q-grams, so reads are added until there are n candidates
    with S.Filter(genome, m, k) as f:
        while have < n:
            r = _reads(case, genome, m, part, seed + 7919 * len(reads))
            for strand in (0, 4):
                c = f.run(r, strand, 1 << 30)
                ids.append(c.ids + base)
                pos.append(c.pos)
                dirs.append(c.dirs)
                have += len(c.ids)
            reads.append(r)
            base += part
    return (np.concatenate(reads), np.concatenate(ids)[:n], np.concatenate(pos)[:n],
            np.concatenate(dirs)[:n])


_COMP = torch.arange(256, dtype=torch.uint8)
for _a, _b in zip(b"ACGT", b"TGCA"):
    _COMP[_a] = _b


def _call_arrays(genome, reads, ids, pos, dirs, m: int, k: int) -> dict:
    """The call layout on the device: windows and reads back to back,
    inclusive offsets, flags."""
    T = lambda a, t: torch.from_numpy(np.ascontiguousarray(a)).cuda().to(t)  # noqa: E731
    g, r, d = T(genome, torch.uint8), T(reads, torch.uint8), T(dirs, torch.int8)
    ids, pos = T(ids, torch.int64), T(pos, torch.int64)
    fl = (d & 3).long()
    length = m + k * ((fl >= 2).long() + (fl % 2))
    goff = torch.cumsum(length, 0)
    n, total = len(d), int(goff[-1])
    at = torch.repeat_interleave(pos - (goff - length), length, output_size=total)
    at += torch.arange(total, device="cuda")
    windows = g[at]
    rd = r[ids]
    rev = d > 3
    rd[rev] = _COMP.cuda()[rd[rev].flip(1).long()]
    pad = torch.zeros(64, dtype=torch.uint8, device="cuda")
    return dict(genome=torch.cat([windows, pad]), reads=torch.cat([rd.reshape(-1), pad]),
                goff=goff.to(torch.int32),
                roff=(torch.arange(1, n + 1, device="cuda") * m).to(torch.int32), dirs=d,
                n=n, bytes=total, slots=total + k * n)


def _zeros(n: int, dtype=torch.uint8, device="cuda"):
    return torch.zeros(n, dtype=dtype, device=device)


def _outputs(m: int, k: int, n: int, compact: bool = False) -> dict:
    """Output buffers with room for the longest windows."""
    o = dict(scores=_zeros(n, torch.int32))
    if compact:
        return dict(o, records=_zeros(n * S.compact_record_bytes(m, k)))
    return dict(o, read_aln=_zeros(n * (m + 3 * k)), genome_aln=_zeros(n * (m + 3 * k)))


def _batch(a: dict, m: int, k: int, c0: int = 0, c1: int | None = None, g0: int = 0,
           g1: int | None = None, goff=None) -> S.SaruBatch:
    c1 = a["n"] if c1 is None else c1
    g1 = a["bytes"] if g1 is None else g1
    goff = a["goff"] if goff is None else goff
    return S.SaruBatch(a["genome"].data_ptr() + g0, a["reads"].data_ptr() + c0 * m,
                       goff.data_ptr() + 4 * c0, a["roff"].data_ptr(), a["dirs"].data_ptr() + c0,
                       c1 - c0, k, 0, 1, 1, m, g1 - g0, g1 - g0 + k * (c1 - c0))


def _lengths(case: dict) -> list[tuple[int, int]]:
    return [(int(x), case["k"] or W.k_for(int(x))) for x in case["lengths"].split(",")]


def _prepare_multi(case: dict, seed: int) -> Kept:
    genome = _genome(case, seed)
    bins, out, batches, results, keep = _lengths(case), {}, [], [], []
    status = _zeros(1, torch.int32)
    for i, (m, k) in enumerate(bins):
        a = _call_arrays(genome, *_candidates(case, genome, m, k, case["n"], seed + 31 * i), m, k)
        n, rb = a["n"], S.compact_record_bytes(m, k)
        o = _outputs(m, k, n, case["compact"])
        # calls at the queue threshold, each with offsets of its own
        step = min(W.chunk_value_for(m, k), max(1, n // 2))
        ends = a["goff"].long().cpu().numpy()
        goff = a["goff"].clone()
        for c0 in range(0, n, step):
            c1 = min(n, c0 + step)
            g0, g1 = int(ends[c0 - 1]) if c0 else 0, int(ends[c1 - 1])
            goff[c0:c1] -= g0
            batches.append(_batch(a, m, k, c0, c1, g0, g1, goff))
            s0 = g0 + k * c0
            sc = o["scores"].data_ptr() + 4 * c0
            if case["compact"]:
                results.append(S.SaruResult(sc, o["records"].data_ptr() + c0 * rb, None,
                                            status.data_ptr()))
            else:
                results.append(S.SaruResult(sc, o["read_aln"].data_ptr() + s0,
                                            o["genome_aln"].data_ptr() + s0, status.data_ptr()))
        keep += [a, goff]
        out[str(m)] = o
    out["status"] = status
    size = S.multi_scratch_bytes(batches)
    return Kept(case=case, batches=batches, results=results, out=out, keep=keep,
                scratch=torch.empty(size, dtype=torch.uint8, device="cuda"))


def prepare(case: dict, seed: int) -> Kept:
    kind = case["kind"]
    if kind == "multi":
        return _prepare_multi(case, seed)
    genome = _genome(case, seed)
    lib = S.load()
    if kind == "filter":
        reads = _reads(case, genome, case["m"], case["reads"], seed + 1)
        most = _most(case, case["reads"])
        out = {x: dict(counts=np.zeros(3, np.int64), call_begin=np.zeros(4096, np.int64),
                       ids=np.zeros(most, np.int32), pos=np.zeros(most, np.int32),
                       dirs=np.zeros(most, np.int8), perfect_ids=np.zeros(most, np.int32),
                       perfect_pos=np.zeros(most, np.int32)) for x in ("0", "4")}
        return Kept(case=case, reads=reads, out=out, most=most,
                    chunk=W.chunk_value_for(case["m"], case["k"]),
                    filter=lib.saru_filter_create(genome.ctypes.data, len(genome), case["m"],
                                                  case["k"], -1))
    if kind == "server":
        bins = _lengths(case)
        per = case["reads"] // len(bins)
        reads = [_reads(case, genome, m, per, seed + i) for i, (m, _) in enumerate(bins)]
        sets = (S.SaruReadSet * len(bins))(*[S.SaruReadSet(r.ctypes.data, per, m, k, 0)
                                             for r, (m, k) in zip(reads, bins)])
        out, most = {}, _most(case, per)
        for m, k in bins:
            o = dict(counts=np.zeros(3, np.int64), ids=np.zeros(most, np.int32),
                     pos=np.zeros(most, np.int32), dirs=np.zeros(most, np.int8),
                     scores=np.zeros(most, np.int32), perfect_ids=np.zeros(most, np.int32),
                     perfect_pos=np.zeros(most, np.int32))
            if case["compact"]:
                o["records"] = np.zeros(most * S.compact_record_bytes(m, k), np.uint8)
            else:
                o["read_aln"] = np.zeros(most * (m + 3 * k), np.uint8)
                o["genome_aln"] = np.zeros(most * (m + 3 * k), np.uint8)
            out[str(m)] = o
        cfg = S.ServerConfig(torch.cuda.current_device(), 1, 64, 2, 4 << 30, 256 << 20)
        server = lib.saru_server_create(C.byref(cfg))
        if lib.saru_server_set_genome(server, genome.ctypes.data, len(genome)):
            raise RuntimeError(S.last_error())
        return Kept(case=case, server=server, sets=sets, keep=reads, out=out, most=most)
    m, k = case["m"], case["k"]
    a = _call_arrays(genome, *_candidates(case, genome, m, k, case["n"], seed), m, k)
    if kind == "device":
        o = dict(_outputs(m, k, a["n"]), status=_zeros(1, torch.int32))
        size = S.scratch_bytes(a["n"], m, k)
        return Kept(case=case, keep=a, out=o, batch=_batch(a, m, k),
                    result=S.SaruResult(o["scores"].data_ptr(), o["read_aln"].data_ptr(),
                                        o["genome_aln"].data_ptr(), o["status"].data_ptr()),
                    scratch=torch.empty(size, dtype=torch.uint8, device="cuda"))
    pin = lambda t: t.cpu().pin_memory()  # noqa: E731
    host = {x: pin(a[x]) for x in ("genome", "reads", "goff", "roff", "dirs")}
    n = a["n"]
    b = W.Batch(m=m, k=k, genome=host["genome"].numpy()[:a["bytes"]],
                reads=host["reads"].numpy()[:n * m], genome_offsets=host["goff"].numpy(),
                read_offsets=host["roff"].numpy(), edit_offsets=np.zeros(0, np.int32),
                dirs=host["dirs"].numpy(), ids=np.zeros(0, np.int32), pos=np.zeros(0, np.int32))
    o = [pin(x) for x in _outputs(m, k, n).values()]
    return Kept(case=case, batch=b, keep=[host, o], out=S.AlignResult(*[x.numpy() for x in o]))


def run(state: Kept):
    kind = state.case["kind"]
    if kind == "device":
        S.align_device(state.batch, state.result, state.scratch.data_ptr(),
                       state.scratch.numel(), torch.cuda.current_stream().cuda_stream)
        return state.out
    if kind == "multi":
        align = S.align_multi_device_compact if state.case["compact"] else S.align_multi_device
        align(state.batches, state.results, state.out["status"].data_ptr(),
              state.scratch.data_ptr(), state.scratch.numel(),
              torch.cuda.current_stream().cuda_stream)
        return state.out
    if kind == "host":
        S.align_host(state.batch, out=state.out)
        return dict(scores=state.out.scores, read_aln=state.out.read_aln,
                    genome_aln=state.out.genome_aln)
    lib = S.load()
    if kind == "filter":
        for strand in (0, 4):
            o = state.out[str(strand)]
            P = {x: a.ctypes.data for x, a in o.items()}
            rc = lib.saru_filter_run(state.filter, state.reads.ctypes.data, len(state.reads),
                                     strand, state.chunk, P["counts"])
            if rc or o["counts"][1:].max() > state.most or o["counts"][0] > 4095:
                raise RuntimeError(f"filter: {rc} {o['counts']} {S.last_error()}")
            lib.saru_filter_results(state.filter, P["call_begin"], P["ids"], P["pos"], P["dirs"],
                                    P["perfect_ids"], P["perfect_pos"])
        return state.out
    ticket, stats, r = C.c_int64(), S.RequestStats(), S.SaruReadResults()
    n = len(state.sets)
    if (lib.saru_server_submit_reads(state.server, state.sets, n, int(state.case["compact"]),
                                     C.byref(ticket))
            or lib.saru_server_wait(state.server, ticket.value, 60_000, C.byref(stats))):
        raise RuntimeError(S.last_error())
    for i, o in enumerate(state.out.values()):
        lib.saru_server_read_results(state.server, ticket.value, i, C.byref(r))
        if r.n > state.most or r.nperfect > state.most:
            raise RuntimeError(f"{r.n} candidates, {r.nperfect} perfect hits")
        o["counts"][:] = r.ncalls, r.n, r.nperfect
        slots = C.cast(r.slot_begin, C.POINTER(C.c_int64))[r.ncalls] if r.ncalls else 0
        for x, a in o.items():
            if x != "counts":
                size = (slots if x.endswith("_aln") else r.n * r.record_bytes if x == "records"
                        else (r.nperfect if x.startswith("perfect") else r.n) * a.itemsize)
                if size:
                    C.memmove(a.ctypes.data, getattr(r, x), size)
    lib.saru_server_release(state.server, ticket.value)
    return state.out


def work(case: dict) -> dict:
    """Bytes of one pass: reads, windows, 9 bytes of offsets and flag in; a
    score and two slots (or a record) out.  The arithmetic is whole-number
    dynamic programming, so there are no floating-point operations."""
    def align(m: int, k: int, n: int, compact: bool = False) -> float:
        window = m + 1.55 * k
        out = S.compact_record_bytes(m, k) if compact else 2 * (window + k)
        return n * (m + window + 13 + out)

    kind = case["kind"]
    if kind == "multi":
        return dict(bytes=sum(align(m, k, case["n"], case["compact"]) for m, k in _lengths(case)),
                    flops=0)
    if kind == "filter":
        # reads in; read id, position and flag of every candidate out
        return dict(bytes=case["reads"] * (case["m"] + 9 * PER_READ[case["genome"]]), flops=0)
    if kind == "server":
        per = case["reads"] // len(_lengths(case))
        return dict(bytes=sum(per * m + align(m, k, int(per * PER_READ[case["genome"]]),
                                              case["compact"])
                              for m, k in _lengths(case)), flops=0)
    return dict(bytes=align(case["m"], case["k"], case["n"]), flops=0)
