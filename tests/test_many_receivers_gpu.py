"""Recorded runs with more receivers than the loop kernel's sampling warps or one
sampling launch's first blocks take: the same rows on every path, and no slower
than sampling launches of their own."""

import statistics

import numpy as np
import pytest

import cases as CS
from casebuild import build_product

pytestmark = pytest.mark.gpu


def _sims(*tunings, **config):
    from ionosphere_fdtd_b200.engine import Tuning

    case = dict(CS.CASES["config1_s2"], init=(3, 1.0e-6))
    case["config"] = dict(case["config"], **config)
    return [build_product(case, "float32", tuning=Tuning(**t)) for t in tunings]


def _receivers(sim, rows):
    rng = np.random.default_rng(rows)
    shape = (rows, 3)
    return (rng.integers(sim.er.shape[0], size=shape), np.broadcast_to(rng.integers(sim.hr.shape[1], size=(rows, 1)), shape),
            np.full(shape, 1.0 / 3.0))


@pytest.mark.parametrize("rows", [1184, 1185, 2000])  # 8 per SM, one more, and more than 512 warps
def test_rows_equal_on_every_path(rows):
    auto, ring, direct = sims = _sims({}, dict(staging=2), dict(staging=1))
    v, k, w = _receivers(auto, rows)
    traces = [sim.record_er_observations(v, k[:, 0], w, 45) for sim in sims]
    h = [sim.record_h_observations(v, k, w, v, k, w, 9, sample_every=2) for sim in sims]
    for other in (1, 2):
        np.testing.assert_array_equal(traces[0], traces[other])
        for a, b in zip(h[0], h[other]):
            np.testing.assert_array_equal(a, b)
    assert np.abs(traces[0]).max() > 0.0
    for f in ("er", "et", "hr", "ht"):
        for other in (ring, direct):
            np.testing.assert_array_equal(auto.to_numpy(getattr(auto, f)), other.to_numpy(getattr(other, f)), err_msg=f)


def _us_per_step(fn, steps):
    import torch

    times = []
    for _ in range(7):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        b.synchronize()
        times.append(1e3 * a.elapsed_time(b) / steps)
    return statistics.median(times)


@pytest.mark.parametrize("level,cells", [(5, 24), (6, 50)])
def test_a_row_for_every_vertex_costs_a_sampling_launch(level, cells):
    """A sampled step against the step and a sampling launch of its own (which has a
    warp per row), with half of both to spare."""

    import torch

    auto, ring = _sims({}, dict(staging=2), subdivision=level, radial_cells=cells)
    steps = 64
    for sim in (auto, ring):
        index = np.stack([(np.arange(sim.er.shape[0]) + i) % sim.er.shape[0] for i in range(3)], axis=1)
        probe = sim._engine.probe("er", index, np.full(index.shape, cells // 2), np.full(index.shape, 1.0 / 3.0))
        out = torch.zeros((steps, probe.rows), dtype=torch.float64, device="cuda")
        state, zero = sim._state(), np.zeros(steps)

        def samples():
            for row in out:
                sim._engine.sample(state, probe, row)

        for _ in range(2):
            sim._engine.step_sampled(state, zero, steps, probe, out)
        sampled = _us_per_step(lambda: sim._engine.step_sampled(state, zero, steps, probe, out), steps)
        step = _us_per_step(lambda: ring._engine.step(ring._state(), zero, steps), steps)
        sample = _us_per_step(samples, steps)
        probe.close()
        assert sampled < 1.5 * (step + sample), (level, sampled, step, sample)


def test_a_plan_gives_large_sample_rows_back():
    """32 steps of 300,000 rows are 77 MB of staging: gone with the run's probe."""

    import torch

    (sim,) = _sims(dict(staging=2))
    v, k, w = _receivers(sim, 300_000)
    first = sim.record_er_observations(v[:8], k[:8, 0], w[:8], 40)
    before = torch.cuda.mem_get_info()[0]
    probe = sim._engine.probe("er", v, k, w)
    out = torch.zeros((32, len(v)), dtype=torch.float64, device="cuda")
    taken = torch.cuda.mem_get_info()[0]
    sim._engine.step_sampled(sim._state(), None, 32, probe, out)
    torch.cuda.synchronize()
    assert taken - torch.cuda.mem_get_info()[0] > 60e6
    probe.close()
    held = out.numel() * 8 + 4e6
    assert before - torch.cuda.mem_get_info()[0] < held + 20e6
    again = sim.record_er_observations(v[:8], k[:8, 0], w[:8], 40)  # the plan's graphs, on new staging
    assert np.isfinite(first).all() and np.abs(again).max() > 0.0
