"""The launch count of a bench line follows the kernel that runs the steps."""

import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.parametrize("steps,rows,loop,launches", [
    (1000, 8, (256, 1184), 4), (256, 1184, (256, 1184), 1), (257, 8, (256, 1184), 2), (100, 1185, (256, 1184), 300), (100, 256, (0, 0), 300)])
def test_launches_of_a_recorded_run(steps, rows, loop, launches):
    sys.path.insert(0, str(ROOT))
    import bench

    assert bench.step_launches(steps, rows, loop) == launches


def test_a_fused_step_is_one_launch_and_its_sampling():
    sys.path.insert(0, str(ROOT))
    import bench

    assert bench.step_launches(100, 8, (0, 0), fused=True) == 200
