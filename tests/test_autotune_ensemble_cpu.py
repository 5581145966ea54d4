"""An ensemble's tuner times candidates in the batched launches that the ensemble
runs: alone, a small member's automatic plan would be timed in another kernel."""

from types import SimpleNamespace

from ionosphere_fdtd_b200 import autotune as A
from ionosphere_fdtd_b200.engine import Tuning
from ionosphere_fdtd_b200.errors import BackendUnavailableError


def _member(cells):
    backend = SimpleNamespace(synchronize=lambda: None, _engine=None, itemsize=4)
    sim = SimpleNamespace(backend=backend, config=SimpleNamespace(subdivision=2, radial_cells=cells), _plasma_coupler=None,
                          _surface_impedance_ade=None, mesh=SimpleNamespace(n_vertices=162))
    sim._engine = backend._engine = SimpleNamespace(tuning=Tuning(), close=lambda: None)
    return sim


def test_candidates_are_timed_as_the_ensemble_runs_them(monkeypatch):
    alone = {1: 2.0, 2: 1.0, 3: 3.0}
    together = {1: 2.0, 3: 1.0}

    def in_batch(sim, engine, steps, repeats):
        if engine.tuning.producer_warps == 2:
            raise BackendUnavailableError("cannot join a batch")
        return together[engine.tuning.producer_warps]

    monkeypatch.setattr(A, "_engine_for", lambda sim, t: SimpleNamespace(tuning=t, close=lambda: None))
    monkeypatch.setattr(A, "_time_engine", lambda sim, engine, steps, repeats: alone[engine.tuning.producer_warps])
    monkeypatch.setattr(A, "_time_in_batch", in_batch, raising=False)
    monkeypatch.setattr(A, "_snapshot", lambda sim: {})
    monkeypatch.setattr(A, "_restore", lambda sim, saved: None)
    members, candidates = [_member(10), _member(10)], [Tuning(producer_warps=n) for n in (1, 2, 3)]
    (res,) = A.autotune_ensemble(members, candidates).values()
    assert res.best.producer_warps == 3 and res.best_ms == 1.0
    assert [err for t, ms, err in res.timings if t.producer_warps == 2] == ["cannot join a batch"]
    assert all(m._engine.tuning.producer_warps == 3 for m in members)
    # a single simulation is still timed on its own
    assert A.autotune(_member(10), candidates).best.producer_warps == 2
