"""The bytes that bench.py credits a kernel with, against the DRAM traffic that
was counted for it: the profile has a row for every kernel of a step, and a
kernel is not credited with bytes that it does not move."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


@pytest.mark.parametrize("kernel", ["sweep_x", "sweep_y", "sweep_z", "ct", "combine", "boundary"])
def test_credited_bytes_were_counted(kernel):
    counted = bench.dram_traffic_table()[kernel]
    # the sweeps' stores can stay in L2 (126 MB) and count with the kernel after: 6 % at 160^3
    assert bench.algorithmic_bytes(kernel, 256, 256, 256) <= 1.07 * counted


def test_combine_is_credited_with_37_arrays():
    n = 64
    arrays = bench.algorithmic_bytes("combine", n, n, n) / (8.0 * (n + 1) ** 3)
    # in: 15 fluxes, 5 of the old state, 3 face fields, and 0, 5, 5 of the current one;
    # out: 8 of the primitives, and 1, 1, 6 of the state
    assert arrays == pytest.approx(23 + 10 / 3 + 8 + 8 / 3)
