"""Performance cases: what users of this framework have it do, over the range they do it in.

A case names one call of the public API: a time-step run of ``GeodesicFDTD`` (plain stepping, a monitored
run, recorded receivers, recorded H samples), an ``Ensemble`` of uneven members, or the trace surrogate's
prediction and training.  ``listed`` gives the standing cases, ``draw`` more of the same ranges, ``prepare``
what a program holds before the call, ``run`` the call, ``work`` the bytes and operations it cannot do
without and ``exact`` the same results from plain float64 torch.
"""

import functools
import math

import numpy as np
import torch

from ionosphere_fdtd_b200 import (
    ELECTRON_MASS_KG,
    ELEMENTARY_CHARGE_C,
    ColdPlasmaSpecies,
    ConductiveHalfSpaceSurface,
    EarthIonosphereMaterial,
    Ensemble,
    GaussianCurrent,
    GeodesicFDTD,
    MeshPlasmaModel,
    SimulationConfig,
    SphericalAnomaly,
    SphericalRefinementRegion,
    build_adaptive_geodesic_mesh,
    build_geodesic_mesh,
)
from ionosphere_fdtd_b200.surrogate import TraceSurrogate, architecture
from ionosphere_fdtd_b200.workloads import (
    ProfileMaterial,
    config3_draws,
    drude_profile_plasma,
    seed_fields,
    smooth_log_normal,
    synthetic_provenance,
    uniform_receivers,
    vertex_lat_lon,
)

DEVICE = "cuda"
EPSILON_0, MU_0 = 8.8541878128e-12, 1.256637062120e-6
OXYGEN_MASS_KG = 16.0 * 1.66053906660e-27


# ---- the cases -------------------------------------------------------------


def _fdtd(name, call, level, cells, steps, *, plasma="none", surface=False, material="profile", receivers=0,
          dtype="float32", mesh="uniform"):
    return {"name": name, "call": call, "level": level, "cells": cells, "steps": steps, "plasma": plasma,
            "surface": surface, "material": material, "receivers": receivers, "dtype": dtype, "mesh": mesh}


def listed():
    return [
        # the smallest call: a program that couples to the solver and advances it one step at a time
        _fdtd("one_step_s3", "step", 3, 24, 1),
        # a whole small run, as in a tutorial or a parameter check: 1,000 steps with 8 surface receivers
        _fdtd("short_run_s2", "record", 2, 24, 1000, receivers=8),
        # magnetic-field stations sampled after every step, ground impedance below
        _fdtd("h_stations_s4", "record_h", 4, 31, 64, surface=True, receivers=12),
        # stepping with the field maxima looked at every 100 steps, volume ground, an odd radial grid
        _fdtd("monitored_s5", "monitor", 5, 37, 100),
        # a locally refined mesh (vertex degree up to 8) around the source, horizontally varying ground,
        # magnetised electrons and ions: the anisotropic plasma with per-face coefficients
        _fdtd("refined_magnetised", "record", 4, 33, 50, plasma="magnetised", material="patchy", receivers=16,
              mesh="refined"),
        # the float64 engine on the full physics: what a convergence or drift study runs
        _fdtd("float64_s5", "record", 5, 40, 50, plasma="drude", surface=True, receivers=16, dtype="float64"),
        # ELF propagation at a moderate resolution: impedance ground, Drude plasma, 32 receivers
        _fdtd("waveguide_s6", "record", 6, 50, 100, plasma="drude", surface=True, receivers=32),
        # the single-run workload: Drude plasma over volume ground, 64 receivers
        _fdtd("drude_s7", "record", 7, 40, 100, plasma="drude", receivers=64),
        # the high-resolution workload: impedance ground, Drude plasma, 256 receivers, state far above L2
        _fdtd("waveguide_s8", "record", 8, 80, 20, plasma="drude", surface=True, receivers=256),
        # an ensemble of uneven members (mesh levels 5 to 7, 24 to 60 radial cells), 16 receivers each
        {"name": "ensemble", "call": "ensemble", "members": 8, "layout": 20260803, "steps": 50, "receivers": 16},
        # the trained surrogate answering a batch of parameter sets
        {"name": "surrogate_predict", "call": "predict", "traces": 4096, "batch": 512, "width": 512, "depth": 4},
        # the surrogate in training
        {"name": "surrogate_fit", "call": "fit", "traces": 2048, "batch": 512, "width": 512, "depth": 4,
         "iterations": 8},
    ]


def draw(rng):
    kind = rng.choice(("fdtd",) * 9 + ("ensemble", "predict", "fit"))
    if kind == "ensemble":
        return {"call": "ensemble", "members": rng.randint(2, 8), "layout": rng.randrange(1 << 30),
                "steps": _log_int(rng, 8, 60), "receivers": rng.randint(1, 24)}
    if kind == "predict":
        return {"call": "predict", "traces": _log_int(rng, 1, 8192), "batch": 512, "width": rng.choice((256, 512)),
                "depth": rng.randint(3, 5)}
    if kind == "fit":
        return {"call": "fit", "traces": _log_int(rng, 600, 4096), "batch": rng.choice((128, 256, 300, 512)),
                "width": rng.choice((256, 512)), "depth": rng.randint(3, 5), "iterations": rng.randint(2, 8)}
    level, cells = rng.randint(2, 7), _log_int(rng, 10, 80)
    plasma = rng.choice(("none", "none", "drude", "drude", "magnetised"))
    mesh = "refined" if level in (3, 4) and rng.random() < 0.3 else "uniform"
    if plasma == "magnetised":
        level = min(level, 5)
    dtype = "float64" if rng.random() < 0.2 else "float32"
    call = rng.choice(("step", "record", "record", "record_h", "monitor"))
    cost = 10 * 4**level * cells * (2 if dtype == "float64" else 1)  # cells of one step, float32 equivalents
    most = max(1, min(400, int(5e8 / cost)))
    case = _fdtd("", call, level, cells, _log_int(rng, 1, most if call != "record_h" else min(most, 100)),
                 plasma=plasma, surface=rng.random() < 0.4,
                 material="patchy" if level <= 5 and rng.random() < 0.2 else "profile",
                 receivers=_log_int(rng, 1, 256) if call.startswith("record") else 0, dtype=dtype, mesh=mesh)
    del case["name"]
    return case


def _log_int(rng, low, high):
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


# ---- what a program holds before the call ------------------------------------


@functools.lru_cache(maxsize=None)
def _mesh(level, kind="uniform"):
    if kind == "refined":
        return build_adaptive_geodesic_mesh(level, (SphericalRefinementRegion(35.0, 126.0, 15.0, level + 2, 20.0),))
    return build_geodesic_mesh(level)


def _magnetised(mesh, mids):
    """A dipole field and electrons with O+ ions whose density follows the latitude."""

    c = np.asarray(mesh.face_centers)
    b = 3.0e-5 * (np.array([0.0, 0.0, 1.0]) - 3.0 * c[:, 2:3] * c)
    shape = (mesh.n_faces, len(mids))
    magnetic = np.ascontiguousarray(np.broadcast_to(b[:, None, :], (*shape, 3)))
    lat = 1.0 + 0.3 * c[:, 2:3]
    density = lat * (1.0e6 * np.exp((mids - 85_000.0) / 3_000.0))[None, :]
    nu = np.broadcast_to(1.0e7 * np.exp(-(mids - 70_000.0) / 6_000.0), shape)
    species = (
        ColdPlasmaSpecies("electron", -ELEMENTARY_CHARGE_C, ELECTRON_MASS_KG, density, nu),
        ColdPlasmaSpecies("O+", ELEMENTARY_CHARGE_C, OXYGEN_MASS_KG, 0.5 * density, 0.02 * nu),
    )
    return MeshPlasmaModel.from_mesh(mesh, mids, magnetic, species, provenance=(synthetic_provenance(),),
                                     interpolation="face centres")


@functools.lru_cache(maxsize=None)
def _plasma(level, kind, cells, bottom, plasma):
    mesh = _mesh(level, kind)
    alt = np.linspace(bottom, 100_000.0, cells + 1)
    # as the solver derives them from the radii
    radii = 6_370_000.0 + alt
    mids = 0.5 * (radii[:-1] + radii[1:]) - 6_370_000.0
    return drude_profile_plasma(mesh, mids) if plasma == "drude" else _magnetised(mesh, mids)


def _simulation(case, seed):
    mesh = _mesh(case["level"], case["mesh"])
    bottom = 0.0 if case["surface"] else -100_000.0
    cfg = SimulationConfig(subdivision=case["level"], radial_cells=case["cells"], minimum_altitude_m=bottom,
                           maximum_altitude_m=100_000.0, earth_radius_m=6_370_000.0,
                           radial_boundary_condition="surface-impedance" if case["surface"] else "pec")
    rng = np.random.default_rng(seed)
    lat, lon = vertex_lat_lon(mesh.vertices, int(rng.integers(mesh.n_vertices)))
    if case["material"] == "patchy":
        material = EarthIonosphereMaterial(anomalies=(
            SphericalAnomaly(30.0, 100.0, 2.5e6, -60_000.0, -1.0, 30.0),
            SphericalAnomaly(-20.0, -50.0, 4.0e6, 55_000.0, 90_000.0, 0.5)))
    else:
        material = ProfileMaterial()
    sim = GeodesicFDTD(
        cfg, material=material,
        source=GaussianCurrent(latitude_deg=lat, longitude_deg=lon, peak_current_a=1.0, carrier_frequency_hz=20.0),
        surface_impedance=ConductiveHalfSpaceSurface(smooth_log_normal(mesh.edge_midpoints(), 20260814)) if case["surface"] else None,
        plasma=None if case["plasma"] == "none" else _plasma(case["level"], case["mesh"], case["cells"], bottom, case["plasma"]),
        mesh=mesh, device=DEVICE, dtype=case["dtype"])
    seed_fields(sim, seed=seed)
    return sim


def _h_samples(mesh, cells, count, seed):
    rng = np.random.default_rng(seed)
    faces, edges = rng.integers(mesh.n_faces, size=(count, 1)), rng.integers(mesh.n_edges, size=(count, 3))
    return (faces, rng.integers(cells, size=(count, 1)), np.ones((count, 1)),
            edges, rng.integers(cells + 1, size=(count, 3)), rng.uniform(0.2, 0.5, (count, 3)))


def _ensemble_members(case, seed):
    """Members of the ensemble configuration: sizes from the case, physics and sources from the seed too."""

    out = []
    draws = config3_draws(seed=case["layout"], members=case["members"])
    for i, (d, p) in enumerate(zip(draws, config3_draws(seed=seed, members=case["members"]))):
        mesh = _mesh(d["subdivision"])
        material = EarthIonosphereMaterial(
            lithosphere_conductivity_s_m=p["ground"], ionosphere_reference_height_m=p["h0"],
            ionosphere_scale_height_m=p["zeta"], ionosphere_prefactor_hz=p["sigma0"] / EPSILON_0)
        lat, lon = vertex_lat_lon(mesh.vertices, p["source_draw"] % mesh.n_vertices)
        sim = GeodesicFDTD(
            SimulationConfig(subdivision=d["subdivision"], radial_cells=d["radial_cells"]), material=material,
            source=GaussianCurrent(latitude_deg=lat, longitude_deg=lon, peak_current_a=1.0, carrier_frequency_hz=p["carrier"]),
            mesh=mesh, device=DEVICE, dtype="float32")
        seed_fields(sim, seed=seed + i)
        out.append((sim, uniform_receivers(sim, case["receivers"], p["receiver_seed"])))
    return out


def _surrogate(case, seed):
    net = TraceSurrogate(architecture(width=case["width"], depth=case["depth"]), seed=seed, device=DEVICE)
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    for b in net.b:
        b.copy_(0.05 * torch.randn(b.shape, generator=g, device=DEVICE))
    n = case["traces"]
    x = (2.0 * torch.rand((n, 8), generator=g, device=DEVICE) - 1.0).to(torch.bfloat16)
    # pulses of the shape the solver's receivers record: one or two lobes per trace
    t = torch.linspace(0.0, 1.0, 1024, device=DEVICE)
    u = torch.rand((n, 4), generator=g, device=DEVICE)
    z = (t[None] - 0.3 - 0.4 * u[:, 0:1]) / (0.05 + 0.1 * u[:, 1:2])
    y = (0.2 + u[:, 2:3]) * (1.0 - 2.0 * u[:, 3:4] * z**2) * torch.exp(-(z**2))
    return net, x, y.contiguous()


def prepare(case, seed):
    call = case["call"]
    if call == "ensemble":
        members = _ensemble_members(case, seed)
        return {"case": case, "ensemble": Ensemble([s for s, _ in members]), "observations": [r for _, r in members]}
    if call in ("predict", "fit"):
        net, x, y = _surrogate(case, seed)
        return {"case": case, "net": net, "x": x, "y": y, "seed": seed}
    sim = _simulation(case, seed)
    state = {"case": case, "sim": sim}
    if call == "record":
        state["receivers"] = uniform_receivers(sim, case["receivers"], seed)
    elif call == "record_h":
        state["samples"] = _h_samples(sim.mesh, case["cells"], case["receivers"], seed)
    return state


# ---- the call ----------------------------------------------------------------


def _state_of(sim):
    out = {"er": sim.er, "et": sim.et, "hr": sim.hr, "ht": sim.ht}
    if sim._plasma_coupler is not None:
        for i, j in enumerate(sim._plasma_coupler.ade.current_density):
            out["j%d" % i] = j
    if sim._surface_impedance_ade is not None:
        out["memory"] = sim._surface_impedance_ade.memory
    return out


def run(state):
    case = state["case"]
    call, steps = case["call"], case.get("steps")
    if call == "ensemble":
        ens = state["ensemble"]
        traces = ens.record_er_observations(state["observations"], steps)
        # 4 fields and the traces of each member
        return [[s.er, s.et, s.hr, s.ht, t] for s, t in zip(ens.members, traces)]
    if call == "predict":
        return state["net"].predict(state["x"], batch=case["batch"])
    if call == "fit":
        net = state["net"]
        losses = net.fit(state["x"], state["y"], iterations=case["iterations"], batch=case["batch"], lr=2e-3, lr_final=2e-5,
                         seed=state["seed"], relative=True)
        return {"losses": losses, "w": net.w, "b": net.b}
    sim = state["sim"]
    out = {}
    if call == "record":
        out["traces"] = sim.record_er_observations(*state["receivers"], steps)
    elif call == "record_h":
        out["hr_samples"], out["ht_samples"] = sim.record_h_observations(*state["samples"], steps)
    else:
        sim.step(steps)
        if call == "monitor":
            d = sim.diagnostics()
            out["maxima"] = [d["max_abs_er_v_m"], d["max_abs_et_v_m"], d["max_abs_hr_a_m"], d["max_abs_ht_a_m"]]
    out.update(_state_of(sim))
    return out


# ---- the work it cannot do without -------------------------------------------


def _step_work(mesh, cells, species, surface, item):
    """One leapfrog step: every state array read once and written once; the stencil's operations."""

    v, e, f, n = mesh.n_vertices, mesh.n_edges, mesh.n_faces, cells
    values = (v + e) * (n + 1) + (e + f) * n + 3 * species * f * n + (16 * e if surface else 0)
    flops = e * (n + 1) * 9 + f * n * 8 + v * (n + 1) * 16 + e * n * 9 + (64 * e if surface else 0)
    if species:
        flops += f * n * (26 + 9 * species) + v * (n + 1) * 40 + e * n * 14
    return 2 * item * values, flops


def _layer_shapes(case, rows):
    width, depth = case["width"], case["depth"]
    shapes = [(rows, 8, width)] + [(rows, width, width)] * (depth - 1) + [(rows, width, 1024)]
    return shapes + [(rows * 16, 64, 128), (rows * 64, 32, 64), (rows * 256, 16, 4)]


def work(case):
    call = case["call"]
    if call == "ensemble":
        b = o = 0
        for d in config3_draws(seed=case["layout"], members=case["members"]):
            x, y = _step_work(_mesh(d["subdivision"]), d["radial_cells"], 0, False, 4)
            b, o = b + x * case["steps"], o + y * case["steps"]
        return {"bytes": b, "flops": o}
    if call in ("predict", "fit"):
        weights = sum(k * n + n for _, k, n in _layer_shapes(case, 1))
        if call == "predict":
            rows = case["traces"]
            return {"bytes": 2 * weights + rows * (16 + 4096), "flops": sum(2 * m * k * n for m, k, n in _layer_shapes(case, rows))}
        rows = min(case["batch"], case["traces"])
        flops = sum(6 * m * k * n for m, k, n in _layer_shapes(case, rows)) - 2 * rows * 8 * case["width"]
        # targets and inputs of the batch; master weights, two moments read and written, bf16 copies written
        return {"bytes": case["iterations"] * (rows * (16 + 4096) + weights * 26), "flops": case["iterations"] * flops}
    species = {"none": 0, "drude": 1, "magnetised": 2}[case["plasma"]]
    b, o = _step_work(_mesh(case["level"], case["mesh"]), case["cells"], species, case["surface"],
                      8 if case["dtype"] == "float64" else 4)
    return {"bytes": b * case["steps"], "flops": o * case["steps"]}


# ---- the same results in float64, from plain torch ----------------------------


class _Exact:
    """The leapfrog step on float64 tensors, from a simulation's mesh tables, material samples and fields."""

    def __init__(self, sim):
        m, self.dt = sim.mesh, float(sim.time_step_s)
        d = lambda a: torch.as_tensor(np.array(a, dtype=np.float64), device=DEVICE)  # noqa: E731
        i = lambda a: torch.as_tensor(np.array(a, dtype=np.int64), device=DEVICE)  # noqa: E731
        self.tail, self.head = i(m.edges[:, 0]), i(m.edges[:, 1])
        self.left, self.right = i(m.edge_left_faces), i(m.edge_right_faces)
        self.faces, self.face_edges = i(m.faces), i(m.face_edges)
        theta, self.phi = d(m.primal_edge_angles), d(m.dual_edge_angles)
        self.inv_theta = 1.0 / theta[:, None]
        area = d(m.face_solid_angles)
        self.circ = d(m.face_edge_signs) * theta[self.face_edges] / area[:, None]
        self.dual_area = d(m.dual_cell_solid_angles)
        self.r = d(sim.radii_m)
        self.mid, self.dr = 0.5 * (self.r[:-1] + self.r[1:]), self.r[1:] - self.r[:-1]
        one = lambda a: a[:1] if np.array_equal(a, np.broadcast_to(a[:1], a.shape)) else a  # noqa: E731
        self.ca_er, self.cb_er = self._loss(d(one(sim.sigma_er)), EPSILON_0 * d(one(sim.epsilon_r_er)))
        self.ca_et, self.cb_et = self._loss(d(one(sim.sigma_et)), EPSILON_0 * d(one(sim.epsilon_r_et)))
        self.source, self.n = sim.source, sim.steps
        v, k, w = sim.source.staggered_distribution(sim)
        self.sv, self.sk = i(v), i(k)
        control = torch.cat((0.5 * self.dr[:1], self.mid[1:] - self.mid[:-1], 0.5 * self.dr[-1:]))
        self.sw = (d(w) * sim.source.vertical_element_length_m / self.dual_area[self.sv] / self.r[self.sk] ** 2 / control[self.sk]
                   * self.cb_er.expand(m.n_vertices, -1)[self.sv, self.sk])
        self.er, self.et, self.hr, self.ht = (getattr(sim, f).double().clone() for f in ("er", "et", "hr", "ht"))
        self.surface = sim.surface_impedance
        if self.surface is not None:
            s = self.surface
            lo = math.log(2 * math.pi * s.minimum_frequency_hz) - s.pole_span_decades * math.log(10.0)
            hi = math.log(2 * math.pi * s.maximum_frequency_hz) + s.pole_span_decades * math.log(10.0)
            pole = torch.exp(lo + (torch.arange(s.terms, device=DEVICE, dtype=torch.float64) + 0.5) * (hi - lo) / s.terms)
            a = 0.5 * self.dt * pole
            self.decay, self.drive = (1 - a) / (1 + a), a / (1 + a)
            self.history = (hi - lo) / s.terms * torch.sqrt(pole) / math.pi / (1 + a)
            self.scale = torch.sqrt(MU_0 / d(s.conductivity_s_m))
            self.memory = torch.zeros((m.n_edges, s.terms), device=DEVICE, dtype=torch.float64)
        self.plasma = sim.plasma
        if self.plasma is not None:
            c = self.centre = d(m.face_centers)
            p = d(m.vertices)
            normal = torch.linalg.cross(p[self.tail], p[self.head])
            normal = normal / normal.norm(dim=1, keepdim=True)
            t = torch.linalg.cross(normal[self.face_edges], c[:, None, :].expand(-1, 3, -1))
            t = t / t.norm(dim=2, keepdim=True)
            # the tangents span the plane normal to the centre: their pseudo-inverse from a full-rank 3 x 3 inverse
            g = t.transpose(1, 2) @ t + c[:, :, None] * c[:, None, :] / (c * c).sum(1)[:, None, None]
            self.recon = (torch.linalg.inv(g) @ t.transpose(1, 2)).transpose(1, 2)
            edge = torch.arange(m.n_edges, device=DEVICE)
            slot = lambda f: (self.face_edges[f] == edge[:, None]).int().argmax(1)  # noqa: E731
            self.t_left, self.t_right = t[self.left, slot(self.left)], t[self.right, slot(self.right)]
            self.vertex_area = torch.zeros(m.n_vertices, device=DEVICE, dtype=torch.float64)
            self.face_area = area
            for q in range(3):
                self.vertex_area.index_add_(0, self.faces[:, q], area)
            row = lambda a: d(a[:1] if a.strides[0] == 0 else a)  # noqa: E731
            b = row(self.plasma.magnetic_field_t)
            size = b.norm(dim=2, keepdim=True)
            self.b = torch.where(size > 0, b / torch.where(size > 0, size, torch.ones_like(size)), torch.zeros_like(b))
            self.coef, self.j = [], []
            for s in self.plasma.species:
                nu, gyro = row(s.collision_frequency_hz), s.charge_c * size[..., 0] / s.mass_kg
                nu, gyro = torch.broadcast_tensors(nu, gyro)
                push = row(s.number_density_m3) * s.charge_c**2 / s.mass_kg
                # integral of exp((-nu + i gyro) t) over the step
                ex, an, den = torch.exp(-nu * self.dt), gyro * self.dt, nu**2 + gyro**2
                u, w = torch.expm1(-nu * self.dt) + ex * (torch.cos(an) - 1.0), ex * torch.sin(an)
                self.coef.append([x[..., None] for x in (ex, torch.cos(an), torch.sin(an), push * -torch.expm1(-nu * self.dt) / nu,
                                                         push * (-nu * u + gyro * w) / den, push * (-nu * w - gyro * u) / den)])
                self.j.append(torch.zeros((m.n_faces, len(self.mid), 3), device=DEVICE, dtype=torch.float64))

    def _loss(self, sigma, eps):
        rate = sigma * self.dt / eps
        phi = torch.where(rate != 0, -torch.expm1(-rate) / torch.where(rate != 0, rate, torch.ones_like(rate)), torch.ones_like(rate))
        return torch.exp(-rate), self.dt / eps * phi

    def magnetic(self):
        k = self.dt / MU_0
        grad = (self.er[self.head] - self.er[self.tail]) * self.inv_theta / self.r
        scaled = self.et * self.mid
        diff = torch.cat((2 * scaled[:, :1] / self.dr[0], (scaled[:, 1:] - scaled[:, :-1]) / (self.mid[1:] - self.mid[:-1]),
                          -2 * scaled[:, -1:] / self.dr[-1]), 1) / self.r
        old = self.ht[:, 0].clone()
        self.ht += k * (grad - diff)
        if self.surface is not None:
            kap = 2 * self.dt / (MU_0 * self.dr[0])
            c = kap * self.scale * self.history.sum()
            past = self.scale * (self.memory @ self.history)
            new = ((1 - 0.5 * c) * old + k * grad[:, 0] - kap * self.mid[0] / self.r[0] * self.et[:, 0] + kap * past) / (1 + 0.5 * c)
            self.memory = self.memory * self.decay + (new + old)[:, None] * self.drive
            self.ht[:, 0] = new
        for q in range(3):
            self.hr -= k / self.mid * self.circ[:, q, None] * self.et[self.face_edges[:, q]]

    def _currents(self):
        nodes = (self.er[self.faces[:, 0]] + self.er[self.faces[:, 1]] + self.er[self.faces[:, 2]]) / 3.0
        e = (0.5 * (nodes[:, 1:] + nodes[:, :-1]))[..., None] * self.centre[:, None, :]
        for q in range(3):
            e += self.et[self.face_edges[:, q]][..., None] * self.recon[:, q, None, :]
        magnetised = bool((self.b != 0).any())
        total = torch.zeros_like(e)
        if magnetised:
            along = (e * self.b).sum(-1, keepdim=True) * self.b
            across = e - along
            turned = torch.linalg.cross(across, self.b.expand_as(e))
        for n, (decay, cos, sin, par, re, im) in enumerate(self.coef):
            j = self.j[n]
            if magnetised:
                ja = (j * self.b).sum(-1, keepdim=True) * self.b
                jc = j - ja
                j = (decay * ja + par * along + decay * (cos * jc + sin * torch.linalg.cross(jc, self.b.expand_as(j)))
                     + re * across + im * turned)
            else:
                j = decay * j + re * e
            self.j[n] = j
            total += j
        radial = (total * self.centre[:, None, :]).sum(2) * self.face_area[:, None]
        at = torch.zeros((self.er.shape[0], radial.shape[1]), device=DEVICE, dtype=torch.float64)
        for q in range(3):
            at.index_add_(0, self.faces[:, q], radial)
        at /= self.vertex_area[:, None]
        jr = torch.cat((at[:, :1], 0.5 * (at[:, 1:] + at[:, :-1]), at[:, -1:]), 1)
        jt = 0.5 * ((total[self.left] * self.t_left[:, None, :]).sum(2) + (total[self.right] * self.t_right[:, None, :]).sum(2))
        return jr, jt

    def electric(self, current):
        jr, jt = self._currents() if self.plasma is not None else (0.0, 0.0)
        flux = self.ht * self.phi[:, None]
        curl = torch.zeros_like(self.er).index_add_(0, self.tail, flux).index_add_(0, self.head, -flux) / self.dual_area[:, None] / self.r
        self.er = self.ca_er * self.er + self.cb_er * (curl - jr)
        self.er.index_put_((self.sv, self.sk), -self.sw * current, accumulate=True)
        scaled = self.ht * self.r
        curl = (self.hr[self.left] - self.hr[self.right]) / self.phi[:, None] / self.mid - (scaled[:, 1:] - scaled[:, :-1]) / self.dr / self.mid
        self.et = self.ca_et * self.et + self.cb_et * (curl - jt)

    def step(self):
        s = self.source
        width = 0.5 / s.carrier_frequency_hz
        t = (self.n + 0.5) * self.dt - max(4.0 * width, 36.0 * self.dt)
        self.magnetic()
        self.electric(s.peak_current_a * math.exp(-((t / width) ** 2)) * math.cos(2 * math.pi * s.carrier_frequency_hz * t))
        self.n += 1

    def outputs(self):
        out = {"er": self.er, "et": self.et, "hr": self.hr, "ht": self.ht}
        if self.plasma is not None:
            out.update({"j%d" % i: j for i, j in enumerate(self.j)})
        if self.surface is not None:
            out["memory"] = self.memory
        return out


def _weighted(field, rows, layers, weights):
    i = lambda a: torch.as_tensor(np.asarray(a), device=DEVICE)  # noqa: E731
    return (field[i(rows), i(layers)] * i(weights)).sum(1)


def _exact_record(sim, receivers, steps):
    x = _Exact(sim)
    v, k, w = receivers
    traces = [_weighted(x.er, v, k[:, None].repeat(v.shape[1], 1), w)]
    for _ in range(steps):
        x.step()
        traces.append(_weighted(x.er, v, k[:, None].repeat(v.shape[1], 1), w))
    return x, torch.stack(traces)


def _exact_net(net, x):
    """Every layer's input and pre-activation, in float64 from the float32 weights."""

    a, kept = x.double(), []
    for i, layer in enumerate(net.layers):
        z = a @ net.w[i].double().T + net.b[i].double()
        kept.append((a, z))
        a = torch.nn.functional.silu(z) if layer.act else z
        a = a.reshape(a.shape[0] * layer.expand, -1) if i + 1 < len(net.layers) else a
    return kept, a.reshape(x.shape[0], -1)


def _exact_fit(net, x, y, seed, case):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    w = [t.double().requires_grad_() for t in net.w]
    b = [t.double().requires_grad_() for t in net.b]
    weight = (1.0 / y.pow(2).mean(dim=1).clamp_min(1e-12 * float(y.pow(2).mean()))).double()
    first, second = [torch.zeros_like(t) for t in w + b], [torch.zeros_like(t) for t in w + b]
    losses = []
    for it in range(case["iterations"]):
        idx = torch.randint(0, len(x), (min(case["batch"], len(x)),), device=DEVICE, generator=gen)
        a = x[idx].double()
        for i, layer in enumerate(net.layers):
            a = a @ w[i].T + b[i]
            a = torch.nn.functional.silu(a) if layer.act else a
            a = a.reshape(a.shape[0] * layer.expand, -1) if i + 1 < len(net.layers) else a
        loss = (weight[idx, None] * (a.reshape(len(idx), -1) - y[idx].double()) ** 2).mean()
        losses.append(float(loss.detach()))
        rate = 2e-3 * (2e-5 / 2e-3) ** (it / max(case["iterations"] - 1, 1))
        with torch.no_grad():
            for p, g, m, v in zip(w + b, torch.autograd.grad(loss, w + b), first, second):
                m.mul_(0.9).add_(0.1 * g)
                v.mul_(0.999).add_(0.001 * g * g)
                p -= rate * (m / (1 - 0.9 ** (it + 1))) / ((v / (1 - 0.999 ** (it + 1))).sqrt() + 1e-8)
    return {"losses": losses, "w": [t.detach() for t in w], "b": [t.detach() for t in b]}


def exact(case, seed):
    state, call = prepare(case, seed), case["call"]
    if call == "ensemble":
        out = []
        for sim, obs in zip(state["ensemble"].members, state["observations"]):
            x, traces = _exact_record(sim, obs, case["steps"])
            out.append([x.er, x.et, x.hr, x.ht, traces])
        return out
    if call == "predict":
        return _exact_net(state["net"], state["x"])[1]
    if call == "fit":
        return _exact_fit(state["net"], state["x"], state["y"], seed, case)
    sim = state["sim"]
    out = {}
    if call == "record":
        x, out["traces"] = _exact_record(sim, state["receivers"], case["steps"])
    else:
        x = _Exact(sim)
        faces, face_layers, fw, edges, edge_layers, ew = state.get("samples") or (None,) * 6
        hr, ht = [], []
        for n in range(case["steps"] + 1):
            if n:
                x.step()
            if call == "record_h":
                hr.append(_weighted(x.hr, faces, face_layers, fw))
                ht.append(_weighted(x.ht, edges, edge_layers, ew))
        if call == "record_h":
            out["hr_samples"], out["ht_samples"] = torch.stack(hr), torch.stack(ht)
        elif call == "monitor":
            out["maxima"] = [float(f.abs().max()) for f in (x.er, x.et, x.hr, x.ht)]
    out.update(x.outputs())
    return out
