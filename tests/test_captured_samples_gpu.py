"""Sampled steps and loop launches inside a caller's captured graph.

A replay must read nothing that the call left behind on the host or that a later
recorded run of the plan moves: between two replays a run with more receivers
takes the plan's sample buffers.
"""

import numpy as np
import pytest

import cases as CS
from casebuild import build_product

pytestmark = pytest.mark.gpu

TUNINGS = [dict(), dict(staging=2), dict(staging=1), dict(fused_step=1)]


def _pair(tuning):
    from ionosphere_fdtd_b200.engine import Tuning

    sims = [build_product(dict(CS.CASES["config1_s2"], init=(3, 1.0e-6)), "float32", tuning=Tuning(**tuning)) for _ in range(2)]
    for sim in sims:
        sim.source = None
        sim.step(40)
    return sims


def _probe(sim, kind, rows, seed):
    rng = np.random.default_rng(seed)
    field = getattr(sim, kind)
    shape = (rows, 3)
    return sim._engine.probe(kind, rng.integers(field.shape[0], size=shape), rng.integers(field.shape[1], size=shape), rng.standard_normal(shape))


def _capture(fn):
    import torch

    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        fn()
    return graph


def _use_the_stack(depth=40):
    return np.random.default_rng(depth).standard_normal(64).sum() + (_use_the_stack(depth - 1) if depth else 0.0)


@pytest.mark.parametrize("tuning", TUNINGS, ids=str)
@pytest.mark.parametrize("every", [1, 2])
def test_captured_sampled_steps_replay(tuning, every):
    import torch

    steps, kinds = 6, ("er", "ht")
    captured, plain = _pair(tuning)
    probes = [[_probe(sim, kind, 11, 5) for kind in kinds] for sim in (captured, plain)]
    outs = [[torch.zeros((steps // every, 11), dtype=torch.float64, device="cuda") for _ in kinds] for _ in range(2)]

    def run(sim, which):
        if every == 1:
            for p, o in zip(probes[which], outs[which]):
                sim._engine.step_sampled(sim._state(), None, steps, p, o)
        else:
            sim._engine.step_recorded(sim._state(), None, steps, every, probes[which], outs[which])

    graph = _capture(lambda: run(captured, 0))
    for replay in range(3):
        graph.replay()
        run(plain, 1)
        _use_the_stack()
        for a, b in zip(*outs):
            assert torch.equal(a, b) and float(a.abs().max()) > 0.0
        for sim in (captured, plain):  # a recorded run of more rows and whole chunks
            more = _probe(sim, "er", 700 * (replay + 1), 9)
            rows = torch.zeros((64, more.rows), dtype=torch.float64, device="cuda")
            sim._engine.step_sampled(sim._state(), None, 64, more, rows)
            more.close()
    torch.cuda.synchronize()
    for f in ("er", "et", "hr", "ht"):
        np.testing.assert_array_equal(captured.to_numpy(getattr(captured, f)), plain.to_numpy(getattr(plain, f)), err_msg=f)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("name", ["config1_s2", "plasma_magnetized_s1", "config4_mini_s2"])
def test_captured_loop_steps_replay(name, dtype):
    import torch

    from ionosphere_fdtd_b200.engine import Tuning

    case = dict(CS.CASES[name], init=(3, 1.0e-6))
    loop, ring = build_product(case, dtype), build_product(case, dtype, tuning=Tuning(staging=2))
    for sim in (loop, ring):
        sim.source = None
        sim.step(2)
    graph = _capture(lambda: loop.step(3))
    for _ in range(4):  # the same calls on both: a Drude current is turned into face frames and back around each
        graph.replay()
        ring.step(3)
    torch.cuda.synchronize()
    for f in ("er", "et", "hr", "ht"):
        np.testing.assert_array_equal(loop.to_numpy(getattr(loop, f)), ring.to_numpy(getattr(ring, f)), err_msg=f)
    assert loop._engine.status_word() == 0
