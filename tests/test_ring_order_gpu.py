"""Ring launches overlap the drain of the launch before them on the stream.

Whatever runs on the stream before or between them (another library's kernels on
the fields, a probe, a captured run, a second plan of an ensemble) must still be seen
whole: the fields equal those of the direct launches, bit for bit.
"""

import numpy as np
import pytest

import cases as CS
from casebuild import build_product

pytestmark = pytest.mark.gpu


def _pair(name, dtype):
    from ionosphere_fdtd_b200.engine import Tuning

    case = dict(CS.CASES[name], init=(3, 1.0e-6))
    return [build_product(case, dtype, tuning=Tuning(staging=s)) for s in (2, 1)]


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("name", ["config1_s2", "plasma_drude_s2", "plasma_magnetized_s1", "surface_map_s2"])
def test_foreign_kernels_between_steps(name, dtype):
    import torch

    ring, direct = _pair(name, dtype)
    for sim in (ring, direct):
        side = torch.cuda.Stream()
        for i in range(12):
            sim.step(1 + i % 3)
            for f in (sim.er, sim.et, sim.hr, sim.ht):
                f.mul_(0.75)
            if i == 6:  # the rest of the run on another stream
                side.wait_stream(torch.cuda.current_stream())
                torch.cuda.set_stream(side)
        torch.cuda.synchronize()
        torch.cuda.set_stream(torch.cuda.default_stream())
    for f in ("er", "et", "hr", "ht"):
        np.testing.assert_array_equal(ring.to_numpy(getattr(ring, f)), direct.to_numpy(getattr(direct, f)), err_msg=f)


@pytest.mark.parametrize("steps", [1, 2, 65])
def test_samples_between_phases(steps):
    """A sample sees the step before it and nothing of the one after."""

    ring, direct = _pair("config1_s2", "float32")
    v, k, w = CS.receiver_rows(ring.mesh.n_vertices, ring.altitudes_m, 5, 150)
    np.testing.assert_array_equal(ring.record_er_observations(v, k, w, steps), direct.record_er_observations(v, k, w, steps))


def test_captured_ring_steps():
    import torch

    ring, direct = _pair("config1_s2", "float32")
    ring.source = direct.source = None
    ring.step(3)
    direct.step(3)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ring.step(2)
    for _ in range(3):
        graph.replay()
    direct.step(6)
    torch.cuda.synchronize()
    for f in ("er", "et", "hr", "ht"):
        np.testing.assert_array_equal(ring.to_numpy(getattr(ring, f)), direct.to_numpy(getattr(direct, f)), err_msg=f)
