"""The exact full-rectangle path where its fill changes form: reads of 6 and 7
bases (the shortest that take the shared-memory rows), matrices that begin at
every place of a 16-byte block, costs whose cells leave 16 bits, reads of
mixed lengths, and reads too long for the rows.  Scores and slots equal the
oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import refkit as R
import saruman_b200 as S
from saruman_b200 import workloads as W

# read length, k, candidates, error rate, alphabet, match, mismatch, flags
CASES = {
    "short6": (6, 2, 200, 0.2, b"ACGT", 0, 1, (1, 2, 3, 5, 6, 7)),
    "short7": (7, 3, 200, 0.2, b"ACGT", 0, 1, (1, 2, 3, 5, 6, 7)),
    "odd": (37, 13, 333, 0.1, b"ACGT", 0, 1, (0, 1, 2, 3, 4, 5, 6, 7)),
    "costs": (40, 3, 100, 0.1, b"ACGTN", 1, 3, (1, 3, 5, 7)),
    "wrap": (40, 3, 100, 0.1, b"ACGT", 0, 3000, (1, 3)),
    "iupac": (100, 5, 200, 0.05, b"ACGTNRYKMSWBDHV", 0, 1, (1, 2, 3)),
    "long": (2600, 16, 3, 0.004, b"ACGT", 0, 1, (1, 3)),
}


def batch(name):
    m, k, n, err, alpha, mat, mis, flags = CASES[name]
    b = W.random_batch(m, k, n, seed=31 * m + k, err=err, alphabet=alpha, flags=flags)
    b.match, b.mismatch = mat, mis
    return b


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CASES))
def test_exact_path_edges(saru_lib, name):
    b = batch(name)
    s1, ra1, ga1, st = R.oracle_align(b, nthreads=8)
    assert st == 0
    r = S.align_host(b)
    np.testing.assert_array_equal(r.scores, s1)
    assert np.array_equal(r.read_aln, ra1) and np.array_equal(r.genome_aln, ga1)


@pytest.mark.gpu
def test_exact_path_mixed_read_lengths(saru_lib):
    rng = np.random.default_rng(3)
    k, n = 3, 150
    lens = rng.integers(8, 60, n)
    reads = [W.BASES[rng.integers(0, 4, int(x))] for x in lens]
    wins = [np.concatenate([r, W.BASES[rng.integers(0, 4, k)]]) for r in reads]
    b = W.make_batch(60, k, wins, np.concatenate(reads), np.full(n, 1, np.int8))
    b.read_offsets = np.cumsum(lens).astype(np.int32)
    b.edit_offsets = np.concatenate([[0], np.cumsum((lens + 1) * (b.lengths + 1))[:-1]]).astype(
        np.int32)
    s1, ra1, ga1, st = R.oracle_align(b, nthreads=8)
    assert st == 0
    r = S.align_host(b)
    np.testing.assert_array_equal(r.scores, s1)
    assert np.array_equal(r.read_aln, ra1) and np.array_equal(r.genome_aln, ga1)
