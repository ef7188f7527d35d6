"""Host calls of 32 MB and more with fewer than 512k candidates (which run in
slices from page-locked arrays) are checked whole before any result is copied
out: a bad candidate at their end leaves the caller's arrays as they were, with
the error an unsliced call gives, from pageable and from page-locked arrays."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import saruman_b200 as S
from saruman_b200 import workloads as W


def big_call(n: int, m: int = 100, k: int = 5, flags=(1, 2, 3, 5, 6, 7)):
    """n candidates that repeat a small batch (regular, one read length)."""
    b = W.random_batch(m, k, 500, seed=n, flags=flags)
    reps = -(-n // b.n)
    lens = np.tile(b.lengths, reps)[:n]
    wins = [b.genome[e - x:e] for e, x in zip(b.genome_offsets, b.lengths)]
    return W.make_batch(m, k, (wins * reps)[:n], np.tile(b.reads.reshape(-1, m), (reps, 1))[:n],
                        np.tile(b.dirs, reps)[:n]), lens


def call(b, go, ro, record_bytes=None, pinned=False):
    """rc and the output arrays, filled before with 0x5A."""
    import torch
    lib = S.load()
    P = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    slots = int(go[-1]) + b.k * b.n
    rb = record_bytes or 16
    room = max(slots, 0)
    sizes = [4 * b.n] + ([room, room] if record_bytes is None else [rb * b.n])
    ins = [b.genome, b.reads, go, ro, b.dirs]
    outs = [np.full(x, 0x5A, np.uint8) for x in sizes]
    keep = []
    if pinned:
        keep = [torch.from_numpy(np.ascontiguousarray(a)).pin_memory() for a in ins + outs]
        arrays = [t.numpy() for t in keep]
        ins, outs = arrays[:5], arrays[5:]
    sb = S.SaruBatch(*[a.ctypes.data for a in ins], b.n, b.k, 0, 1, 1, b.m, int(go[-1]), slots)
    if record_bytes is None:
        sr = S.SaruResult(*[a.ctypes.data for a in outs], None)
        rc = lib.saru_align_host(C.byref(sb), C.byref(sr), 0)
    else:
        rc = lib.saru_align_host_compact(C.byref(sb), P(outs[0]), P(outs[1]), rb, 0)
    return rc, outs


def spoil(b, what: str):
    """The call's offsets with a bad candidate at 3 before its end."""
    go, ro = b.genome_offsets.copy(), b.read_offsets.copy()
    if what == "window":
        go[-3] = go[-4]
    else:
        ro[-3] = ro[-4] - 1
    return go, ro


@pytest.mark.parametrize("what", ["window", "read"])
def test_a_refused_call_names_the_candidate_without_a_gpu(saru_lib, what):
    import torch
    if torch.cuda.is_available():
        pytest.skip("the check runs before a GPU is looked for only where there is none")
    b, _ = big_call(80_001)
    rc, outs = call(b, *spoil(b, what))
    assert rc == S.SARU_E_INVALID and f"candidate {b.n - 3} has" in S.last_error()
    assert all((o == 0x5A).all() for o in outs)


@pytest.mark.parametrize("at", [0, 1, 2, 1023, 1024, 1025, 2048, 2049, 2998, 2999])
@pytest.mark.parametrize("what", ["empty", "decreasing", "long"])
def test_the_first_bad_candidate_is_named(saru_lib, at, what):
    """At the edges of the blocks the check takes at once, with other lengths
    behind it."""
    b, _ = big_call(3000, m=36, k=2)
    lens = np.diff(b.genome_offsets, prepend=0)
    go, ro = b.genome_offsets.copy(), b.read_offsets.copy()
    if what == "empty":
        ro[at:] -= 36
    elif what == "decreasing":
        go[at:] -= lens[at] + 1
    else:
        go[at:] += 32001
    rc, outs = call(b, go, ro)
    assert rc == S.SARU_E_INVALID and f"candidate {at} has" in S.last_error()
    assert all((o == 0x5A).all() for o in outs)


def test_offsets_that_wrap_32_bits_are_refused(saru_lib):
    """Windows that reach 2^31 bytes and go on from -2^31: the differences of
    the offsets are right in 32 bits."""
    b, _ = big_call(75_000, m=36, k=2)
    lens = np.diff(b.genome_offsets, prepend=0).astype(np.int64)
    lens[:67_105] = 32_000
    ends = np.cumsum(lens)
    assert ends[67_104] < 2**31 < ends[-1] and lens[67_105] < 50
    go = ((ends + 2**31) % 2**32 - 2**31).astype(np.int32)
    assert go[-1] < 0
    rc, _ = call(b, go, b.read_offsets)
    first = int(np.argmax(ends >= 2**31))
    assert rc == S.SARU_E_INVALID and f"candidate {first} has" in S.last_error()


@pytest.mark.gpu
@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("n", [80_001, 300_000])
@pytest.mark.parametrize("compact", [False, True])
def test_a_refused_call_leaves_the_outputs(saru_lib, n, pinned, compact):
    b, _ = big_call(n)
    rb = S.compact_record_bytes(b.m, b.k) if compact else None
    for what in ("window", "read"):
        rc, outs = call(b, *spoil(b, what), rb, pinned)
        assert rc == S.SARU_E_INVALID and f"candidate {n - 3} has" in S.last_error()
        assert all((o == 0x5A).all() for o in outs)
    rc, outs = call(b, b.genome_offsets, b.read_offsets, rb, pinned)  # the lane still works
    assert rc == S.SARU_OK
    want = S.align_host(b, lane=1)
    assert np.array_equal(outs[0].view(np.int32), want.scores)
    if compact:
        o = S.expand_compact(b, outs[0].view(np.int32), outs[1], rb)
        assert np.array_equal(o.read_aln, want.read_aln)
        assert np.array_equal(o.genome_aln, want.genome_aln)
    else:
        assert np.array_equal(outs[1], want.read_aln)
        assert np.array_equal(outs[2], want.genome_aln)


@pytest.mark.gpu
@pytest.mark.parametrize("pinned", [False, True])
def test_records_of_an_irregular_call_need_no_more_than_its_strings(saru_lib, pinned):
    """A call that takes the exact path (one window a base too long) accepts
    records that hold its strings but not the longest one possible: windows
    as long as their reads (the last one a base longer), so a string of score k
    has at most (k + 1) / 2 gaps in a read of m bases."""
    b, lens = big_call(300_000, m=40, k=7, flags=(0,))
    rb = S.compact_record_bytes(b.m, b.k) - 16
    assert 4 + 4 * -(-(b.m + (b.k + 1) // 2) // 16) <= rb
    more = lens.copy()
    more[-1] += 1
    go = np.cumsum(more).astype(np.int32)
    b.genome = np.concatenate([b.genome, b.genome[-1:]])
    rc, outs = call(b, go, b.read_offsets, rb, pinned)
    assert rc == S.SARU_OK, S.last_error()
    b.genome_offsets = go
    want = S.align_host(b, lane=1)
    assert np.array_equal(outs[0].view(np.int32), want.scores)
    o = S.expand_compact(b, outs[0].view(np.int32), outs[1], rb)
    assert np.array_equal(o.read_aln, want.read_aln)
