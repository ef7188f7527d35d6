"""Compact records of a launch whose tiles change layout: the bytes of a call
of longer reads, staged while a warp finishes its tile of a call of shorter
ones, reach over that tile's gap masks.  Many short calls of 12 to 40 bases
and different k share one launch of few warps, so that every warp goes from
call to call (last tiles partly filled); scores and records equal the
oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import refkit as R
import saruman_b200 as S
from saruman_b200 import workloads as W

SHAPES = [(40, 0), (16, 4), (36, 0), (12, 3), (40, 7), (20, 5), (24, 7), (13, 2), (36, 2), (33, 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("warps", [1, 4])
def test_compact_records_across_layouts(saru_lib, warps):
    import torch
    dev = torch.device("cuda:0")
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    sbs, crs, keep = [], [], []
    for i in range(190):
        m, k = SHAPES[i % len(SHAPES)]
        b = W.random_batch(m, k, 33 + 7 * i % 190, seed=i, err=0.08,
                           alphabet=b"ACGTN" if i % 7 == 3 else b"ACGT")
        rb = S.compact_record_bytes(m, k)
        t = [T(b.genome), T(b.reads), T(b.genome_offsets), T(b.read_offsets), T(b.dirs),
             torch.zeros(b.n, dtype=torch.int32, device=dev),
             torch.full((b.n * rb,), 0x5A, dtype=torch.uint8, device=dev)]
        keep.append((b, rb, t))
        sbs.append(S.SaruBatch(*[x.data_ptr() for x in t[:5]], b.n, k, 0, 1, 1, m,
                               len(b.genome), b.total_genome))
        crs.append(S.SaruResult(t[5].data_ptr(), t[6].data_ptr(), None, None))
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    try:
        S.set_tuning(40, 7, warps, 1, 0)
        nscr = S.multi_scratch_bytes(sbs)
        scratch = torch.empty(nscr, dtype=torch.uint8, device=dev)
        S.align_multi_device_compact(sbs, crs, status.data_ptr(), scratch.data_ptr(), nscr,
                                     torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
    finally:
        S.clear_tuning()
    assert int(status.item()) == 0
    for b, rb, t in keep:
        s1, ra1, ga1, st = R.oracle_align(b, nthreads=4)
        assert st == 0
        sc = t[5].cpu().numpy()
        np.testing.assert_array_equal(sc, np.minimum(s1, b.k + 1))
        o = S.expand_compact(b, sc, t[6].cpu().numpy(), rb)
        assert np.array_equal(o.read_aln, ra1) and np.array_equal(o.genome_aln, ga1)
