"""CPU check of the diagonal kernel's tile code (diag_tile.cuh): its phases
emulated lane by lane on the host under AddressSanitizer, with the shared
slice and every array exactly sized and the arrays misaligned on purpose;
scores, slot strings and compact records compared with the oracle.  This is
how the kernel's indexing is checked before it runs on a GPU."""
from __future__ import annotations

import ctypes as C
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
SRC = ROOT / "tests" / "harness" / "diag_host.cpp"
SO = ROOT / "tests" / "_build" / "libdiag_host_asan.so"

# read length, k: edges of the 32-column words, of the byte table (255 / 256) and
# of the 32-bit diagonal word (k = 9 / 10), m = 3k + 1, the smallest reads
SHAPES = [(36, 2), (100, 5), (31, 3), (32, 1), (33, 4), (64, 7), (95, 9), (128, 10), (150, 9),
          (250, 15), (255, 12), (46, 15), (2, 0), (8, 1), (40, 13), (16, 5), (256, 12), (300, 9), (512, 15)]


def exact(a: np.ndarray, off: int) -> np.ndarray:
    """Copy of `a` that ends with its allocation, `off` bytes past a 16-byte
    boundary (when the allocator aligns)."""
    raw = np.empty(a.nbytes + off, np.uint8)
    v = raw[off:].view(a.dtype)
    v[...] = a.reshape(-1)
    return v


def compare(lib, m: int, k: int) -> int:
    import refkit as R
    import saruman_b200 as S
    from saruman_b200 import workloads as W
    P = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    bad = 0
    for seed, (err, alpha, flags) in enumerate([
            (0.04, b"ACGT", (1, 2, 3, 5, 6, 7)), (0.1, b"ACGT", (1, 3)),
            (0.3, b"ACGTNR", (1, 2, 3)), (0.05, b"ACGTN", (0, 2, 4, 7)),
            (0.15, b"AC", (1, 2, 3, 5, 6, 7)), (0.02, b"A" * 9 + b"CGT", (1, 2, 3, 6))]):
        n = 193 + 31 * seed
        b = W.random_batch(m, k, n, seed=seed + 97 * m + k, err=err, alphabet=alpha, flags=flags)
        s1, ra1, ga1, _ = R.oracle_align(b, nthreads=4)
        off = (5 * seed + m) % 16
        g, r, d = exact(b.genome, off), exact(b.reads, (off + 5) % 16), exact(b.dirs, 1)
        go, ro = exact(b.genome_offsets, 0), exact(b.read_offsets, 0)
        rb = S.compact_record_bytes(m, k)

        def call(n1, t0, sc, ra, ga, rec):
            return lib.diag_align_batch(
                P(g), P(r), P(go), P(ro), P(d), C.c_long(n1), C.c_int(k), C.c_int(m),
                C.c_int(1 if k <= 9 and m <= 200 and seed % 3 < 2 else 0), C.c_int(1), C.c_long(t0), P(sc), P(ra),
                P(ga), P(rec) if rec is not None else None, C.c_long(rb))
        sc, sl = np.zeros(n, np.int32), np.zeros(b.total_genome, np.uint8)
        ra, ga = exact(sl, (off + 7) % 16), exact(sl, (off + 11) % 16)
        st = call(64, 0, sc, ra, ga, None) | call(n, 64, sc, ra, ga, None)  # in two slices
        want = np.minimum(s1, k + 1)
        if st or not (np.array_equal(want, sc) and np.array_equal(ra1, ra)
                      and np.array_equal(ga1, ga)):
            bad += 1
            print("MISMATCH", m, k, seed, st, np.nonzero(want != sc)[0][:5],
                  np.nonzero(ra1 != ra)[0][:5], np.nonzero(ga1 != ga)[0][:5], flush=True)
        rec = exact(np.zeros(n * rb, np.uint8), 0)
        st = call(n, 0, sc, ra, ga, rec)
        o = S.expand_compact(b, sc, rec, rb, nthreads=2)
        if st or not (np.array_equal(want, sc) and np.array_equal(ra1, o.read_aln)
                      and np.array_equal(ga1, o.genome_aln)):
            bad += 1
            print("COMPACT MISMATCH", m, k, seed, st, flush=True)
    # a window far too long (its tile is not staged) and one a base too long
    b = W.random_batch(m, k, 70, seed=1)
    for more in (100000, 1):
        go = b.genome_offsets.copy()
        go[40:] += more
        g, sl = np.full(int(go[-1]), 65, np.uint8), np.zeros(int(go[-1]) + k * b.n, np.uint8)
        sc, ra, ga = np.zeros(b.n, np.int32), exact(sl, 3), exact(sl, 9)
        st = lib.diag_align_batch(P(g), P(b.reads), P(go), P(b.read_offsets), P(b.dirs),
                                  C.c_long(b.n), C.c_int(k), C.c_int(m), C.c_int(0), C.c_int(1),
                                  C.c_long(0), P(sc), P(ra), P(ga), None, C.c_long(0))
        if not st & 1 or sc[40] != k + 1:
            bad += 1
            print("irregular tile not reported", st, flush=True)
    return bad


@pytest.fixture(scope="module")
def asan_lib():
    SO.parent.mkdir(exist_ok=True)
    csrc = ROOT / "saruman_b200" / "csrc"
    deps = [SRC, csrc / "diag_tile.cuh", csrc / "band_tile.cuh", csrc / "saru_core.cuh"]
    if not SO.exists() or SO.stat().st_mtime < max(d.stat().st_mtime for d in deps):
        subprocess.run(["g++", "-O1", "-g", "-std=c++17", "-shared", "-fPIC",
                        "-fsanitize=address", "-fno-omit-frame-pointer", "-o", str(SO),
                        str(SRC)], check=True)
    return SO


@pytest.mark.parametrize("m,k", SHAPES)
def test_diag_tile_emulation_under_asan(asan_lib, m, k):
    asan = subprocess.run(["gcc", "-print-file-name=libasan.so"], capture_output=True,
                          text=True).stdout.strip()
    env = dict(os.environ, LD_PRELOAD=asan, ASAN_OPTIONS="detect_leaks=0:abort_on_error=0")
    r = subprocess.run([sys.executable, __file__, str(asan_lib), str(m), str(k)],
                       capture_output=True, text=True, env=env, timeout=600)
    assert r.returncode == 0 and "BAD 0" in r.stdout, (r.stdout[-3000:], r.stderr[-3000:])


if __name__ == "__main__":
    sys.path[:0] = [str(ROOT), str(ROOT / "tests")]
    n_bad = compare(C.CDLL(sys.argv[1]), int(sys.argv[2]), int(sys.argv[3]))
    print("BAD", n_bad)
    sys.exit(1 if n_bad else 0)
