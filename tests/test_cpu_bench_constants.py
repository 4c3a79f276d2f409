"""The bench's measured constants belong to the present kernels: FP64 op counts
per point and the V-cycle's DRAM traffic are captures of kernels that change."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

import bench  # noqa: E402


def test_no_group_runs_the_fp64_pipe_above_its_rate():
    # event times of the groups at 512x256x256 on a GB300, ms per launch
    per_launch = {"eno_yz": 0.991, "eno_x": 0.901, "jacobi": 0.765}
    t = bench.group_table({g: (100 * ms, 100) for g, ms in per_launch.items()}, {}, peak_hbm=6780.7, fp64_rate=5.28e11,
                          npts=513 * 257 * 257, ncell=512 * 256 * 256)
    for g in per_launch:
        assert 0.75 < t[g]["fp64_frac"] < 0.95, (g, t[g])


def test_vcycle_traffic_is_spread_over_its_launches():
    # half sweeps, residual, restriction and prolongation of the levels above
    # 32768 cells (4 + 4, 5 + 5 and twice 12 + 12 sweeps), one launch below, two conversions
    launches = sum(4 * n + 3 for n in (4, 5, 12, 12)) + 1 + 2
    assert bench.MG_TRAFFIC_PER_LAUNCH == pytest.approx(7.19e9 / launches)
