"""Launches around the number of tiles up to which warps take them in turn
(four a warp) instead of from a counter: one warp a CTA and one CTA an SM put
that line at 128 candidates an SM.  Scores (k + 1 for any above k) and slots equal
the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import refkit as R
import saruman_b200 as S
from saruman_b200 import workloads as W


@pytest.mark.gpu
@pytest.mark.parametrize("beyond", [-128, -31, 0, 1, 33])
def test_tiles_in_turn_and_from_the_counter(saru_lib, beyond):
    import torch

    n = 128 * torch.cuda.get_device_properties(0).multi_processor_count + beyond
    b = W.random_batch(36, 2, n, seed=n)
    s1, ra1, ga1, st = R.oracle_align(b, nthreads=8)
    assert st == 0
    try:
        S.set_tuning(36, 2, 1, 1, 0)
        r = S.align_host(b)
    finally:
        S.clear_tuning()
    np.testing.assert_array_equal(np.minimum(r.scores, 3), np.minimum(s1, 3))
    assert np.array_equal(r.read_aln, ra1) and np.array_equal(r.genome_aln, ga1)
