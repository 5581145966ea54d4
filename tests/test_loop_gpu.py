"""Many steps in one cooperative launch (``kd_loop``, the automatic plan on small meshes).

The loop kernel runs the step kernels' per-run arithmetic, so its results must
equal those of the ring launches bit for bit: below one run per SM, with a
remainder in the last round, over several rounds, across the 256 steps of one
launch, with every physics branch, and with receivers of each field kind.
"""

import numpy as np
import pytest

import cases as CS
from casebuild import build_product

pytestmark = pytest.mark.gpu

CASES = ["random_s1", "config1_s2", "tangential_s1", "nonuniform_s0", "plasma_drude_s2", "plasma_magnetized_s1", "surface_map_s2",
         "config4_mini_s2", "adaptive_plasma_si_s1"]


def _state(sim) -> dict[str, np.ndarray]:
    out = {f: sim.to_numpy(getattr(sim, f)) for f in ("er", "et", "hr", "ht")}
    if sim._plasma_coupler is not None:
        for i, j in enumerate(sim._plasma_coupler.ade.current_density):
            out[f"plasma_current_{i}"] = sim.to_numpy(j)
    if sim._surface_impedance_ade is not None:
        out["si_memory"] = sim.to_numpy(sim._surface_impedance_ade.memory)
    return out


def _pair(case, dtype):
    """The automatic plan, and the same case on explicitly asked-for ring launches."""

    from ionosphere_fdtd_b200.engine import Tuning

    return build_product(case, dtype), build_product(case, dtype, tuning=Tuning(staging=2))


def _assert_same(a, b):
    ea, eb = _state(a), _state(b)
    for key in ea:
        np.testing.assert_array_equal(ea[key], eb[key], err_msg=key)
    assert a._engine.status_word() == 0


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("name", CASES)
def test_loop_equals_ring_launches_bitwise(name, dtype):
    loop, ring = _pair(CS.CASES[name], dtype)
    for n in (1, 2, 7):
        loop.step(n)
        ring.step(n)
        _assert_same(loop, ring)
    assert np.abs(loop.to_numpy(loop.er)).max() > 0.0


@pytest.mark.parametrize("subdivision,cells,plasma", [(3, 25, False), (5, 37, False), (6, 13, False), (4, 25, True), (5, 25, True)])
def test_loop_rounds_and_remainders(subdivision, cells, plasma):
    """Radial grids off the 16-byte pitch and one to ten rounds of runs."""

    case = dict(CS.CASES["plasma_drude_s2" if plasma else "config1_s2"])
    case["config"] = dict(case["config"], subdivision=subdivision, radial_cells=cells)
    case["init"] = (3, 1.0e-6)
    loop, ring = _pair(case, "float32")
    loop.step(3)
    ring.step(3)
    _assert_same(loop, ring)


@pytest.mark.parametrize("steps", [255, 256, 257, 513])
def test_loop_receivers_across_launches(steps):
    loop, ring = _pair(CS.CASES["config1_s2"], "float32")
    v, k, w = CS.receiver_rows(loop.mesh.n_vertices, loop.altitudes_m, 5, 150)
    np.testing.assert_array_equal(loop.record_er_observations(v, k, w, steps), ring.record_er_observations(v, k, w, steps))
    _assert_same(loop, ring)


@pytest.mark.parametrize("kind", ["er", "et", "hr", "ht"])
def test_loop_samples_every_field_kind(kind):
    import torch

    rng = np.random.default_rng(8)
    loop, ring = _pair(CS.CASES["plasma_drude_s2"], "float32")
    field = getattr(loop, kind)
    index, layer = rng.integers(field.shape[0], size=(9, 37)), rng.integers(field.shape[1], size=(9, 37))
    weight = rng.standard_normal((9, 37))
    rows = []
    for sim in (loop, ring):
        probe = sim._engine.probe(kind, index, layer, weight)
        out = torch.zeros((6, 9), dtype=torch.float64, device="cuda")
        sim._engine.step_sampled(sim._state(), sim._source_currents(6), 6, probe, out)
        rows.append(out.cpu().numpy())
        probe.close()
    np.testing.assert_array_equal(rows[0], rows[1])
    assert np.abs(rows[0]).max() > 0.0


@pytest.mark.parametrize("tuning", [dict(staging=2), dict(staging=2, graph_chunk=4), dict(fused_step=1)], ids=str)
@pytest.mark.parametrize("steps,every", [(9, 1), (9, 2), (64, 7), (300, 128)])
def test_recorded_h_samples_equal_single_steps(steps, every, tuning):
    """One recorded run against stepping to each sample, on the loop and on the
    launched plans (their sampled graph chunks and their steps between samples)."""

    from ionosphere_fdtd_b200.engine import Tuning

    case = CS.CASES["config1_s2"]
    sims = [build_product(case, "float32"), build_product(case, "float32", tuning=Tuning(**tuning))]
    rng = np.random.default_rng(4)
    m, cells = sims[0].mesh, len(sims[0].radii_m) - 1
    faces, edges = rng.integers(m.n_faces, size=(70, 1)), rng.integers(m.n_edges, size=(3, 2))
    args = (faces, rng.integers(cells, size=(70, 1)), np.ones((70, 1)),
            edges, rng.integers(cells + 1, size=(3, 2)), np.full((3, 2), 0.5))
    single = build_product(case, "float32")
    rows = [single.record_h_observations(*args, 0)]
    while single.steps < steps:
        single.step(min(every, steps - single.steps))
        rows.append(single.record_h_observations(*args, 0))
    for sim in sims:
        for n, got in enumerate(sim.record_h_observations(*args, steps, sample_every=every)):
            np.testing.assert_array_equal(got, np.concatenate([r[n] for r in rows]))
        assert sim.steps == steps
        _assert_same(sim, single)
