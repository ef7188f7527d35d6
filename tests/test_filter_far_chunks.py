"""The filter position by position on a genome chunk that begins beyond 2^31
bases (saru_filter_set_chunk takes positions up to 2^32): it keeps what the
step-by-step restatement keeps there, whose ranges are 32-bit positions without
a sign.  CPU only."""
from __future__ import annotations

import subprocess

import pytest

from test_filter_position import exe  # noqa: F401  (fixture)


@pytest.mark.parametrize("m,k", [(36, 2), (100, 5), (24, 5), (150, 9)])
@pytest.mark.parametrize("offset", [2**31, 3_000_000_000, 2**32 - 6100])
def test_positions_beyond_two_gigabases(exe, m, k, offset):  # noqa: F811
    kept = 0
    for unit in (13, 40, 300):
        for seed in range(3):
            r = subprocess.run([str(exe), f"{m},{k},{unit},{offset - 2**32},{seed}"],
                               capture_output=True, text=True)
            assert r.returncode == 0, r.stdout
            kept += int(r.stdout.split()[1])
    assert kept > 100
