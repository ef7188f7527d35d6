"""CPU check of the rows form's columns past a read's end (diag_tile.cuh).

A level's start goes on one column past its neighbours', so on a diagonal that
has reached the window's end column m + e is looked up at level e.  A column
that leaves the diagonal's own row reads the next diagonal's first columns, and
a long match there runs on to columns that do not fit a one-byte cell: read
lengths whose columns m .. m + k cross into another 32-column word are cut at m.
Here every read length up to 200 that crosses, and the ones just below that need
no cut, with reads that hang over the window's end and neighbours that continue
them, against the oracle; the tile code runs under AddressSanitizer and checks
that every stored cell fits its width."""
from __future__ import annotations

import ctypes as C
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "saruman_b200" / "csrc"
HARNESS = {"cut": "diag_host.cpp", "uncut": "diag_host_uncut.cpp"}
BUILD = ROOT / "tests" / "_build"

# two candidates whose read and first window follow; the second window begins
# with the read's last eight bases
READ8 = (b"GATGATATGCCAATCCACAGAAGCGAGGGGGAATTGCCCGAATTCAAATCTCAAGAAGAAGTTTCCCGGGCGCCAGGGCTTCGTATC"
         b"GCAGGGGCCCTGGCATCCCTATTGACGTTTTCGGCTTACCTAGTATGTTAAAGGGCTCGTTCTGCCTTGCT")
WIN8 = (b"GATTTTAGGATGATATGCCAATCCACAGAAGCGAGGGGGAATTGCCCGAATTCAAATCTCAAGAAGAAGTTTCCCGGGCGCCAGGGC"
        b"TTCGTATCGCAGGGGCCCTGGCATCCCTATTGACGTTTTCGGCTTACCTAGTATGCTTAAAGGGCTCGTTCTGCCTT",
        b"GCCTTGCTCCGTCTTATCAGGACAATCCCCGGCCCGTTCCATGGGAATGGGGTAGCGAGTGAGTTCATATGACAAGAGCTGGTTTTT"
        b"AAAAGTTACTCCCCCTCTAGCCTCGTTACAAATCCGAGGTCGACTTACGGCCCTGCTTATTATTGCAAAACGTACAT")
# a read of two letters whose neighbours are runs of G
READ_CA = (b"CCCCACCCACAACCCCCAAAACCACCCACACACACCCCAACACACCAACCAAACACACACAACAAAAACCACCCAAACACCCCAAAA"
           b"ACACCCCAAACCCACCCCAACAACCACACCAACCCACCCACACAAAACACCCAACCAAAACACCAAACAAA")
WIN_CA = (b"AAAGCTTCGCCCCACCCACAACCCCCAAAACCACCCACACACACCCCAACACACCAACCAAACACACACAACAAAAACCACCCAAACA"
          b"CCCCAAAAACACCCCAAACCCACCCCAACAACCACACCAACCCACCCACACAAAACACCCCAACCAAAACACCAAA")


def arr(b: bytes) -> np.ndarray:
    return np.frombuffer(b, np.uint8)


def named_batches():
    from saruman_b200 import workloads as W
    flag = lambda n: np.full(n, 2, np.int8)  # noqa: E731
    yield W.make_batch(158, 6, [arr(w) for w in WIN8], arr(READ8 * 2), flag(2))
    wins = [arr(b"G" * 164), arr(WIN_CA), arr(b"CAA" + b"G" * 161)]
    yield W.make_batch(158, 6, wins, arr(b"G" * 158 + READ_CA + b"G" * 158), flag(3))


def overhanging_batch(m: int, k: int, n: int, seed: int):
    """Reads whose last 0..k bases lie past their window's end: after them the
    next candidate's window goes on with the read (now and then), and the
    reads begin with runs, repeat short units or are random."""
    from saruman_b200 import workloads as W
    rng = np.random.default_rng(seed)
    base = lambda x: W.BASES[rng.integers(0, 4, x)]  # noqa: E731
    flags = rng.choice([1, 2, 3, 5, 6, 7], n, p=[.1, .4, .1, .1, .2, .1]).astype(np.int8)
    wins, reads = [], []
    tail = base(0)
    for f in flags:
        so, eo = W.flank(int(f), k)
        L = m + so + eo
        kind = rng.integers(0, 4)
        if kind == 0:
            r = np.concatenate([np.full(int(rng.integers(m // 3, m - k)), base(1)[0]), base(m)])[:m]
        elif kind == 1:
            r = np.tile(base(int(rng.integers(1, 4))), m)[:m]
        else:
            r = base(m)
        r = r.copy()
        if rng.integers(0, 2):
            r[m - int(rng.integers(1, k + 2)):] = r[0]
        edited = list(r)
        for _ in range(int(rng.integers(0, k + 1))):
            at = int(rng.integers(0, len(edited))) if rng.integers(0, 2) else \
                max(0, len(edited) - 1 - int(rng.integers(0, 12)))
            what = rng.integers(0, 3)
            if what == 0:
                edited[at] = int(base(1)[0])
            elif what == 1:
                edited.insert(at, int(base(1)[0]))
            elif len(edited) > 2:
                del edited[at]
        before = int(rng.integers(0, 2 * k + 1)) if so else int(rng.integers(0, k + 1))
        pre = base(before) if rng.integers(0, 2) else np.full(before, r[0])
        whole = np.concatenate([pre, np.asarray(edited, np.uint8), base(L)])
        w = whole[:L].copy()
        if tail.size and rng.integers(0, 3):  # the window before goes on here
            w[:tail.size] = tail
        over = before + m - L
        tail = r[m - over - int(rng.integers(0, 4)):][:L].copy() if over > 0 else base(0)
        wins.append(w)
        reads.append(r)
    return W.make_batch(m, k, wins, np.concatenate(reads), flags)


def compare(lib, b, rows: int) -> str:
    import refkit as R
    import saruman_b200 as S
    P = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    s1, ra1, ga1, status = R.oracle_align(b, nthreads=4)
    assert status == 0
    rb = S.compact_record_bytes(b.m, b.k)
    sc, rec = np.zeros(b.n, np.int32), np.zeros(b.n * rb, np.uint8)
    ra, ga = np.zeros(b.total_genome, np.uint8), np.zeros(b.total_genome, np.uint8)

    def call(records):
        return lib.diag_align_batch(
            P(b.genome), P(b.reads), P(b.genome_offsets), P(b.read_offsets), P(b.dirs),
            C.c_long(b.n), C.c_int(b.k), C.c_int(b.m), C.c_int(rows), C.c_int(1), C.c_long(0),
            P(sc), P(ra), P(ga), P(rec) if records else None, C.c_long(rb))
    want = np.minimum(s1, b.k + 1)
    st = call(False)
    if st or not np.array_equal(sc, want):
        return f"scores (status {st}, {np.count_nonzero(sc != want)} differ)"
    if not (np.array_equal(ra, ra1) and np.array_equal(ga, ga1)):
        return "slots"
    call(True)
    o = S.expand_compact(b, sc, rec, rb, nthreads=2)
    return "" if np.array_equal(o.read_aln, ra1) and np.array_equal(o.genome_aln, ga1) else "records"


def near(word: int, cut: bool) -> list[tuple[int, int]]:
    """(m, k) of the rows form whose columns m .. m + k cross into column
    32 * word, or (not cut) end just before it or begin just behind it."""
    edge = 32 * word
    if cut:
        shapes = [(m, k) for k in range(2, 10) for m in range(edge - k, edge - 1)]
    else:
        shapes = [(m, k) for k in range(0, 10) for m in (edge - k - 1, edge - 1, edge)]
    return [(m, k) for m, k in shapes if max(2, 3 * k + 1) <= m <= 200]


@pytest.fixture(scope="module")
def asan_lib():
    BUILD.mkdir(exist_ok=True)
    harness = ROOT / "tests" / "harness"
    deps = [*harness.glob("diag_host*.cpp"), CSRC / "diag_tile.cuh", CSRC / "band_tile.cuh",
            CSRC / "saru_core.cuh"]

    def build(form: str) -> Path:
        so = BUILD / f"libdiag_{form}_asan.so"
        if not so.exists() or so.stat().st_mtime < max(d.stat().st_mtime for d in deps):
            subprocess.run(["g++", "-O1", "-g", "-std=c++17", "-shared", "-fPIC",
                            "-fsanitize=address", "-fno-omit-frame-pointer", "-o", str(so),
                            str(harness / HARNESS[form])], check=True)
        return so
    return build


def child(so: Path, form: str, what: str) -> None:
    asan = subprocess.run(["gcc", "-print-file-name=libasan.so"], capture_output=True,
                          text=True).stdout.strip()
    env = dict(os.environ, LD_PRELOAD=asan, ASAN_OPTIONS="detect_leaks=0:abort_on_error=0")
    r = subprocess.run([sys.executable, __file__, str(so), form, what], capture_output=True,
                       text=True, env=env, timeout=900)
    assert r.returncode == 0 and "BAD 0" in r.stdout, (r.stdout[-3000:], r.stderr[-3000:])


def test_reads_over_the_window_end_and_their_neighbours(asan_lib):
    child(asan_lib("cut"), "cut", "named")


@pytest.mark.parametrize("form", ["cut", "uncut"])
@pytest.mark.parametrize("word", [1, 2, 3, 4, 5, 6])
def test_columns_past_the_read(asan_lib, word, form):
    child(asan_lib(form), form, str(word))


@pytest.mark.gpu
@pytest.mark.parametrize("m,k", [(158, 4), (158, 5), (158, 6), (157, 6), (126, 5), (93, 8), (62, 7)])
def test_reads_over_the_window_end_on_the_gpu(saru_lib, m, k):
    import refkit as R
    import saruman_b200 as S
    named = [b for b in named_batches() if (b.m, b.k) == (m, k)]
    for b in named + [overhanging_batch(m, k, 400, seed=7 * m + k)]:
        s1, ra1, ga1, status = R.oracle_align(b, nthreads=4)
        assert status == 0
        r = S.align_host(b)
        np.testing.assert_array_equal(r.scores, np.minimum(s1, k + 1))
        assert np.array_equal(r.read_aln, ra1) and np.array_equal(r.genome_aln, ga1)


def main() -> int:
    lib, cut = C.CDLL(sys.argv[1]), sys.argv[2] == "cut"
    if sys.argv[3] == "named":
        batches = list(named_batches())
    else:
        shapes = near(int(sys.argv[3]), cut)
        assert cut or not any(lib.diag_columns_cross(m, k) for m, k in shapes)
        batches = [overhanging_batch(m, k, 160, seed=1000 * s + 10 * m + k)
                   for m, k in shapes for s in range(3)]
    bad = 0
    for b in batches:
        for rows in (1, 0) if cut else (1,):
            wrong = compare(lib, b, rows)
            if wrong:
                bad += 1
                print("MISMATCH", b.m, b.k, "rows" if rows else "planes", wrong, flush=True)
    print("BAD", bad)
    return 1 if bad else 0


if __name__ == "__main__":
    sys.path[:0] = [str(ROOT), str(ROOT / "tests")]
    sys.exit(main())
