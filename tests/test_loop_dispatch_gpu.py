"""Which plans step in the loop kernel (``kd_loop``): one case on each side of every
line of the rule, the same bits as the direct launches on both sides, and the
explicit geometries, graph chunks and single phases that never use it."""

import numpy as np
import pytest

import cases as CS
from casebuild import build_product, run_product

pytestmark = pytest.mark.gpu


def _state(sim) -> dict[str, np.ndarray]:
    out = {f: sim.to_numpy(getattr(sim, f)) for f in ("er", "et", "hr", "ht")}
    if sim._plasma_coupler is not None:
        for i, j in enumerate(sim._plasma_coupler.ade.current_density):
            out[f"plasma_current_{i}"] = sim.to_numpy(j)
    if sim._surface_impedance_ade is not None:
        out["si_memory"] = sim.to_numpy(sim._surface_impedance_ade.memory)
    return out


# rounds of runs: 148 CTAs of 736 threads (480 with plasma or in float64) against the larger phase's runs
@pytest.mark.parametrize("name,level,cells,dtype,loop", [
    ("config1_s2", 5, 48, "float32", True),  # 5.9 rounds
    ("config1_s2", 5, 51, "float32", False),  # 6.1
    ("config1_s2", 5, 15, "float64", True),  # 5.8
    ("config1_s2", 5, 16, "float64", False),  # 6.6
    ("surface_map_s2", 5, 31, "float32", True),  # 3.8, surface impedance
    ("surface_map_s2", 5, 32, "float32", False),  # 4.04
    ("plasma_magnetized_s1", 5, 50, "float32", True),  # 9.4, magnetised
    ("plasma_magnetized_s1", 5, 64, "float32", False),  # 12.0
    ("config1_s2", 6, 16, "float32", True),  # 8.6, rows of four runs
    ("config1_s2", 6, 17, "float32", False),  # 9.4, rows of five
])
def test_the_lines_of_the_rule(name, level, cells, dtype, loop):
    from ionosphere_fdtd_b200.engine import Tuning

    case = dict(CS.CASES[name])
    case["config"] = dict(case["config"], subdivision=level, radial_cells=cells)
    case["init"] = (3, 1.0e-6)
    auto, direct = build_product(case, dtype), build_product(case, dtype, tuning=Tuning(staging=1))
    assert auto._engine.loop_launch == ((256, 8 * 148) if loop else (0, 0))
    assert direct._engine.loop_launch == (0, 0)
    for n in (1, 3):
        auto.step(n)
        direct.step(n)
    a, b = _state(auto), _state(direct)
    for key in a:
        np.testing.assert_array_equal(a[key], b[key], err_msg=key)
    assert auto._engine.status_word() == 0


@pytest.mark.parametrize("tuning", [dict(staging=1), dict(staging=2), dict(staging=3), dict(graph_chunk=0), dict(producer_warps=1),
                                    dict(e_producer_warps=2), dict(e_threads=256), dict(threads=128), dict(faces_per_patch=32),
                                    dict(e_faces_per_patch=16), dict(lane_layout=2), dict(e_stages=2), dict(fused_step=1)], ids=str)
def test_an_asked_for_geometry_launches_its_phases(tuning):
    from ionosphere_fdtd_b200.engine import Tuning

    assert build_product(CS.CASES["config1_s2"], "float32")._engine.loop_launch[0] == 256
    assert build_product(CS.CASES["config1_s2"], "float32", tuning=Tuning(**tuning))._engine.loop_launch == (0, 0)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("staging", [1, 2])
def test_replayed_chunks_and_direct_launches_agree_bitwise(staging, dtype):
    """Two whole chunks of a captured graph and a remainder, against no graph."""

    from ionosphere_fdtd_b200.engine import Tuning

    case = dict(CS.CASES["config4_mini_s2"], steps=19)
    direct = run_product(case, dtype, tuning=Tuning(staging=staging, graph_chunk=0))
    graphed = run_product(case, dtype, tuning=Tuning(staging=staging, graph_chunk=8))
    for key in ("er", "et", "hr", "ht", "si_memory", "plasma_current_0", "traces"):
        np.testing.assert_array_equal(direct[key], graphed[key], err_msg=key)
