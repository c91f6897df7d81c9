"""The bench's work model: leaves solved pair by pair and by Jacobi sweeps
each count their own work."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402

PAIRS = 16 * (10 * 8 * 15 + 26 * 16 + 4 * 256)  # one leaf, pair by pair
SWEEP = 120 * (12 * 16 + 15)                    # one Jacobi sweep


@pytest.mark.parametrize("sweeps_sum,sweeps_max,jacobi", [(0, 0, 0), (6, 6, 1), (11, 6, 2), (600, 6, 100)])
def test_leaf_work_of_both_kinds(sweeps_sum, sweeps_max, jacobi):
    diag = {"leaf_count": 100, "leaf_sweeps_sum": sweeps_sum, "leaf_sweeps_max": sweeps_max, "level": []}
    work, per = bench.work_model(diag, 0)
    assert per == []
    assert work == (100 - jacobi) * PAIRS + sweeps_sum * SWEEP
