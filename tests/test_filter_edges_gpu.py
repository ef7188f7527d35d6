"""The device filter against its host restatement (pinned to the reference
program's calls by test_filter_host.py) where its layout has edges: more kept
positions in a read than shared memory caches, reads longer than the cached
read, more reads than one launch takes, lists longer than a warp, Ns, and a
genome whose q-grams repeat from position 0 on."""
from __future__ import annotations

import numpy as np
import pytest

import saruman_b200 as S
from saruman_b200 import workloads as W
from test_filter_host import harness, host_calls

pytestmark = pytest.mark.gpu


def tandem(unit: int, copies: int, seed: int, changed: float) -> np.ndarray:
    rng = np.random.default_rng(seed)
    g = np.tile(W.BASES[rng.integers(0, 4, unit)], copies)
    at = rng.random(g.size) < changed
    g[at] = np.frombuffer(b"ACGTN", np.uint8)[rng.integers(0, 5, int(at.sum()))]
    return g


CASES = {
    # m, k, genome, reads, queue threshold
    "kept": (48, 3, lambda: tandem(61, 400, 1, 0.002), 300, 5000),
    "lists": (36, 2, lambda: tandem(40, 700, 2, 0.01), 200, 900),
    "long": (600, 15, lambda: W.uniform_genome(30_000, 3), 120, 40),
    "launches": (36, 2, lambda: W.uniform_genome(20_000, 4), 66_000, 10_000),
    "one": (20, 1, lambda: tandem(25, 60, 5, 0.05), 1, 1),
}


@pytest.mark.parametrize("name", list(CASES))
def test_device_filter_edges(saru_lib, name):
    m, k, genome, nreads, chunk = CASES[name]
    g = genome()
    reads = W.sample_reads(g, nreads, m, 0.02, seed=9).seqs
    lib = harness()
    with S.Filter(g, m, k) as f:
        for dr in (0, 4):
            cb, ids, pos, dirs = host_calls(lib, g, reads, m, k, dr, chunk)
            out = f.run(reads, dr, chunk)
            assert np.array_equal(out.call_begin, cb)
            assert np.array_equal(out.ids, ids)
            assert np.array_equal(out.pos, pos)
            assert np.array_equal(out.dirs, dirs)
            if name == "kept":
                assert np.bincount(out.ids).max() > 96
