"""The work whose speed this repository watches: baking substeps through the public entry points.

``listed()`` names the cases, ``draw(rng)`` gives another of the same ranges. ``prepare`` builds what
a program holds before the call (a simulator, its start state, a batch, captured graphs, a trained
network), ``run`` makes one pass: the start state is put back, then the program's own calls.
``exact`` is the same pass in 64-bit torch, restated from the method (MLS-MPM with quadratic
B-splines, Hencky strain from the matrix logarithm, gradients by autograd), ``work`` the bytes and
operations one pass cannot do without.

A case is a body and what is done with it.

* Bodies. ``loaf``: a box of dough sorted by cell (Ding material, gas, thermal-water transport).
  ``ball``: a dough ball on a fine mesh, a third of whose particles own boundary faces. ``sphere``:
  the same without gas. ``cube``: a tetrahedral cube sampled tet by tet, in sample order, elastic or
  Ding without transport.
* Calls. ``step``: checked substeps one by one (a program that watches every substep). ``advance``:
  many substeps, checked at the end. ``rollout``: forward and backward (calibration). ``batch``:
  many small bodies at once. ``graphs``: one captured substep at a time, new inputs uploaded and a
  result read each time. With ``network`` yielding particles take the learned return map.
"""

from __future__ import annotations

import math
from dataclasses import replace
from functools import lru_cache
from pathlib import Path

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

import baking_b200
from baking_b200.config import DingConfig, MaterialConfig, SimulationConfig
from baking_b200.geometry import BoundaryFaces, CreateDemoMesh, SampleParticles
from baking_b200.scenes import Scene, box_loaf, dough_ball, jittered_sphere, make_simulator

GAS_CONSTANT = 8.31446261815324


# ------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # An interactive viewer or a controller that looks at a small body after every substep: the
        # 64^3 dough sphere of radius 0.1, two launch phases and two flag reads each time.
        dict(name="sphere_9k_step", call="step", body="sphere", grid=64, particles=8_700, steps=4, warm_k=298.0,
             strain=0.0),
        # The same sphere baked headless for a frame's worth of substeps.
        dict(name="sphere_9k_advance", call="advance", body="sphere", grid=64, particles=8_700, steps=40, warm_k=298.0,
             strain=0.0),
        # A neo-Hookean specimen in the reference's own sampling order (four points to a tet of a
        # 12-voxel cube on the default 40^3 grid): mechanics alone.
        dict(name="elastic_cube_41k", call="advance", body="cube", grid=40, particles=41_472, steps=40, warm_k=293.0,
             strain=0.01, material="elastic"),
        # A Ding specimen without transport, five random points to a tet (odd count, ragged order),
        # strained so that it yields: the uncoupled return map.
        dict(name="ding_cube_39k", call="advance", body="cube", grid=40, particles=39_930, steps=40, warm_k=303.0,
             strain=0.06, material="ding"),
        # An ordinary loaf, a fifth of a million particles, about to yield where it is warm.
        dict(name="loaf_201k_advance", call="advance", body="loaf", grid=96, particles=201_417, steps=20, warm_k=309.0,
             strain=0.02),
        # The headline loaf of bench.py: a million particles, elastic.
        dict(name="loaf_1m_advance", call="advance", body="loaf", grid=128, particles=1_000_000, steps=20,
             warm_k=293.15, strain=0.0),
        # The largest scene: four million particles on 256^3, part-baked and pre-stressed, every
        # particle on the plastic branch with the coupled porosity solve.
        dict(name="loaf_4m_yielding", call="advance", body="loaf", grid=256, particles=4_000_000, steps=6,
             warm_k=318.0, strain=0.08),
        # The pre-stressed million-particle loaf with the learned return map.
        dict(name="loaf_1m_network", call="advance", body="loaf", grid=128, particles=1_000_000, steps=20,
             warm_k=318.0, strain=0.08, network=True),
        # Calibration on a small tet-sampled specimen: gradients with respect to the initial
        # velocities and Young's modulus.
        dict(name="rollout_elastic_8k", call="rollout", body="cube", grid=40, particles=8_232, steps=16, every=8,
             warm_k=293.0, strain=0.01, material="elastic"),
        # bench.py's differentiable rollout: a 100k dough ball on 64^3, a checkpoint every 8 substeps.
        dict(name="rollout_ball_100k", call="rollout", body="ball", grid=64, particles=100_000, steps=16, every=8,
             warm_k=330.0, strain=0.04),
        # A bakery sheet: small dough balls of different sizes advanced together.
        dict(name="batch_12_balls", call="batch", body="ball", grid=40, particles=8_000, bodies=12, steps=40,
             warm_k=318.0, strain=0.06),
        # A control loop around the headline loaf: new source rates up and a result down every substep.
        dict(name="loaf_1m_graphs", call="graphs", body="loaf", grid=128, particles=1_000_000, steps=20,
             warm_k=293.15, strain=0.0),
    ]


def draw(rng):
    def size(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high))))) | 1

    def even(low, high):
        return 2 * rng.randint(low // 2, high // 2)

    kind = rng.choice(["loaf", "loaf", "loaf_network", "ball", "sphere", "cube", "rollout_loaf", "rollout_ball",
                       "rollout_cube", "batch", "graphs"])
    warm, strain = rng.choice([(293.15, 0.0), (309.0, 0.02), (318.0, 0.08), (rng.uniform(294.0, 330.0),
                                                                             rng.uniform(0.0, 0.08))])
    case = dict(call="advance", body="loaf", grid=rng.choice([64, 96, 128]), particles=size(60_000, 1_500_000),
                steps=even(6, 20), warm_k=round(warm, 2), strain=round(strain, 4))
    # 12 to 60 particles in each cell of the loaf's 0.012 m^3 (every tet needs one)
    case["particles"] = min(max(case["particles"], 12 * case["grid"] ** 3 * 12 // 1000 | 1),
                            60 * case["grid"] ** 3 * 12 // 1000 | 1)
    if kind == "loaf_network":
        case.update(network=True, warm_k=318.0, strain=round(rng.uniform(0.05, 0.09), 4))
    elif kind in ("ball", "sphere"):
        case.update(body=kind, grid=rng.choice([32, 48, 64]), particles=size(2_000, 120_000), steps=even(8, 40),
                    call=rng.choice(["advance", "advance", "step"]))
        if case["call"] == "step":
            case["steps"] = even(2, 8)
    elif kind == "cube":
        case.update(body="cube", grid=rng.choice([40, 48]), particles=size(2_000, 90_000), steps=even(8, 40),
                    material=rng.choice(["elastic", "ding"]), strain=round(rng.uniform(0.005, 0.06), 4))
    elif kind == "rollout_loaf":
        case.update(call="rollout", grid=64, particles=size(60_000, 180_000), steps=8, every=rng.choice([3, 4, 8]),
                    strain=round(rng.uniform(0.01, 0.08), 4))
    elif kind == "rollout_ball":
        case.update(call="rollout", body="ball", grid=rng.choice([48, 64]), particles=size(5_000, 90_000),
                    steps=even(6, 12), every=rng.choice([4, 8]), strain=round(rng.uniform(0.01, 0.06), 4))
    elif kind == "rollout_cube":
        case.update(call="rollout", body="cube", grid=40, particles=size(2_000, 40_000), steps=even(8, 16),
                    every=rng.choice([4, 8]), material=rng.choice(["elastic", "ding"]),
                    strain=round(rng.uniform(0.005, 0.06), 4))
    elif kind == "batch":
        case.update(call="batch", body="ball", grid=rng.choice([32, 40]), particles=size(3_000, 12_000),
                    bodies=rng.randint(4, 16), steps=even(10, 40), strain=round(rng.uniform(0.0, 0.08), 4))
    elif kind == "graphs":
        case.update(call="graphs")
    return case


# ------------------------------------------------------------------------------------------ scenes
def _cube(case):
    """A 0.3 m cube of tets with the sample count nearest to the case's: 4 (the symmetric rule) or 5
    (random) points to a tet, as the reference's sampler draws them."""
    per_tet = 4 if case["particles"] % 8 in (0, 4) else 5
    voxels = max(2, round((case["particles"] / (6.0 * per_tet)) ** (1.0 / 3.0)))
    mesh = CreateDemoMesh(voxels)
    ding = case["material"] == "ding"
    material = MaterialConfig(model="ding2019" if ding else "neo_hookean")
    simulation = replace(SimulationConfig(), grid_resolution=case["grid"], grid_spacing=1.0 / case["grid"],
                         device_name="cuda:0")
    return Scene("cube", mesh, SampleParticles(mesh, material.density, per_tet), simulation, material,
                 DingConfig(yield_stress=200.0, viscosity=1e6, porosity=0.1) if ding else None, None)


@lru_cache(maxsize=16)
def _body(body, grid, particles, material, warm, seed):
    if body == "cube":
        return _cube(dict(grid=grid, particles=particles, material=material))
    if body == "sphere":
        radius = 0.1 * (particles / 8_751 / (grid / 64) ** 3) ** (1.0 / 3.0)
        return jittered_sphere(grid, 2, min(radius, 0.28), (0.5, 0.5, 0.3 if radius < 0.2 else 0.5), seed)
    if body == "ball":
        return dough_ball(grid, particles, seed, initial_temperature=warm)
    return box_loaf(grid, particles, seed, initial_temperature=warm)


def _scenes(case):
    """The case's scenes. The geometry follows from the case; what changes with the seed is the state."""
    count = case.get("bodies", 1)
    return [_body(case["body"], case["grid"], int(case["particles"] * (0.6 + 0.8 * k / max(1, count - 1)))
                  if count > 1 else case["particles"], case.get("material", "ding"), case["warm_k"], k)
            for k in range(count)]


def _strain(case):
    return np.array([0.5, -1.0, 0.5]) * case["strain"]


def _start(scene, case, seed, index=0):
    """The start state that the seed gives, as float64 tensors holding the values the simulator's
    arrays take: a smooth motion with its velocity gradient, the pre-stretch, temperatures that vary
    smoothly (with a little noise), per-particle gas source rates."""
    rng = np.random.default_rng(1_000_003 * int(seed) + index)
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def f32(a):
        return torch.as_tensor(np.ascontiguousarray(a, np.float32), device=dev)

    x = f32(scene.samples.particle_positions).double()
    n = len(x)
    rates = torch.as_tensor(0.6 * rng.standard_normal((3, 3)), device=dev)
    wave = torch.as_tensor(rng.uniform(8.0, 16.0, 3) * rng.choice([-1.0, 1.0], 3), device=dev)
    push = torch.as_tensor(0.05 * rng.standard_normal(3), device=dev)
    angle = x @ wave + float(rng.uniform(0.0, 6.0))
    centre = x.mean(0)
    v = (x - centre) @ rates.T + torch.sin(angle)[:, None] * push
    C = rates + torch.cos(angle)[:, None, None] * (push[:, None] * wave[None, :])
    stretch = torch.as_tensor(np.diag(np.exp(_strain(case))).astype(np.float32).astype(np.float64), device=dev)
    s = dict(x=x, v=v.float().double(), C=C.float().double(), F=stretch.expand(n, 3, 3).contiguous())
    if scene.material.model == "ding2019":
        s["Fe"] = s["F"].clone()
        s["tau"] = torch.zeros(n, 3, 3, dtype=torch.float64, device=dev)
        s["porosity"] = torch.full((n,), float(np.float32(scene.ding.porosity)), dtype=torch.float64, device=dev)
        s["gelled"] = torch.zeros(n, dtype=torch.int32, device=dev)
        noise = torch.as_tensor(rng.standard_normal(n), device=dev)
        warm = case["warm_k"] + 3.0 * torch.sin(x @ wave.flip(0)) + 0.02 * noise
        if scene.transport is not None:
            volume = torch.as_tensor(scene.samples.reference_volumes, device=dev)
            s["T"] = warm
            s["W"] = scene.transport.water_density * scene.transport.initial_saturation * volume
        else:
            s["T"] = warm.float().double()
        if scene.ding.gas_enabled:
            moles = scene.ding.gas_initial_pressure_pa * scene.ding.porosity / (GAS_CONSTANT * case["warm_k"])
            s["N"] = torch.full((n,), moles, dtype=torch.float64, device=dev)
            s["rate"] = f32(rng.uniform(0.0, 1e-3, n)).double()
    return s


def _arrays(sim):
    """The simulator's primary arrays under the names of ``_start``."""
    st = sim.current_state
    m, t = st.material_state, st.transport_state
    a = dict(x=st.particle_positions, v=st.particle_velocities, C=st.affine_velocities, F=st.deformation_gradients)
    if m is not None:
        a.update(Fe=m.elastic_gradients, tau=m.kirchhoff_stresses, porosity=m.porosities, gelled=m.gelled)
        if sim.material.ding_config.gas_enabled:
            a["N"] = m.gas_moles
        if t is None:
            a["T"] = m.temperatures
    if t is not None:
        a.update(T=t.temperatures, W=t.water_masses)
    return a


def _accumulators(sim):
    t = sim.current_state.transport_state
    return [] if t is None else [t.water_losses, t.heat_exchanges]


# ------------------------------------------------------------------------------------------ a pass
class _Start:
    """A copy of the start state in the arrays' own layout, put back with one call."""

    def __init__(self, sims):
        self.live = [self._flat(t) for s in sims for t in [*_arrays(s).values(), *_accumulators(s)]]
        self.saved = [t.clone() for t in self.live]

    @staticmethod
    def _flat(t):
        planes = t[0].numel()
        return t.as_strided((planes * (t.stride(-1) if planes > 1 else t.shape[0]),), (1,))

    def put_back(self):
        torch._foreach_copy_(self.live, self.saved)


def prepare(case, seed):
    sims, starts = [], []
    for k, scene in enumerate(_scenes(case)):
        s = _start(scene, case, seed, k)
        sim = make_simulator(scene, diagnostics="lean")
        for name, array in _arrays(sim).items():
            array.copy_(s[name])
        if "rate" in s:
            sim.SetGasSourceRates(s["rate"].float().cpu().numpy())
        sims.append(sim)
        starts.append(s)
    state = dict(case=case, sims=sims, start=_Start(sims))
    if case.get("network"):
        from baking_b200.surrogate import LoadReturnSurrogate, ReturnMapSurrogate
        weights = Path(baking_b200.__file__).parent / "data" / "return_surrogate_box_loaf.npz"
        state["network"] = ReturnMapSurrogate(LoadReturnSurrogate(weights)).attach(sims[0])
    if case["call"] == "batch":
        from baking_b200.batch import BatchedSimulators
        state["batch"] = BatchedSimulators(sims).capture()
    elif case["call"] == "graphs":
        from baking_b200.batch import SubstepGraphs
        state["host_rates"] = [_rates(starts[0]["rate"], k).float().cpu().pin_memory() for k in range(case["steps"])]
        state["graphs"] = SubstepGraphs(sims[0], inputs=[sims[0].material.production_parameter],
                                        host_results=True).capture()
        state["copies"] = torch.cuda.Stream()
    elif case["call"] == "rollout":
        s = starts[0]
        state["target"] = _target(s["x"])
        state["inputs"] = {name: value.requires_grad_() for name, value in _differentiated(sims[0], s).items()}
    state["start"].put_back()
    return state


def _rates(rate, k):
    """The source rates a control loop sets before substep k."""
    return (rate * (1.0 + 0.25 * math.sin(0.7 * k))).float().double()


def _target(x):
    """The shape a calibration wants: the initial cloud relaxed from its pre-stretch and grown."""
    centre = x.mean(0)
    return (x - centre) * torch.tensor([1.1, 1.4, 1.1], dtype=x.dtype, device=x.device) + centre


def _differentiated(sim, s):
    if sim.transport is not None:
        return dict(transport_temperatures=s["T"].clone(), gas_source_rates=s["rate"].float(),
                    young_modulus=torch.tensor([2e4], device=s["x"].device))
    return dict(velocities=s["v"].float(), young_modulus=torch.tensor([2e4], device=s["x"].device))


def run(state):
    case, sims = state["case"], state["sims"]
    sim = sims[0]
    state["start"].put_back()
    if case["call"] == "rollout":
        from baking_b200.physics.adjoint import Rollout
        inputs = state["inputs"]
        out = Rollout(sim, case["steps"], checkpoint_every=case["every"], **inputs)
        loss = ((out["positions"].double() - state["target"]) ** 2).sum(1).mean()
        gradients = torch.autograd.grad(loss, list(inputs.values()))
        return dict(state={k: v.detach() for k, v in out.items()}, loss=loss.detach(),
                    gradients=dict(zip(inputs, gradients)))
    if case["call"] == "batch":
        state["batch"].Advance(case["steps"])
        bodies = [_arrays(s) for s in sims]
        return {name: torch.cat([b[name] for b in bodies]) for name in bodies[0]}  # the sheet as one cloud
    if case["call"] == "graphs":
        graphs, results, pending = state["graphs"], [], None
        graphs.load([state["host_rates"][0]], 0, state["copies"])
        for k in range(case["steps"]):
            result = graphs.Advance(1)
            if k + 1 < case["steps"]:
                graphs.load([state["host_rates"][k + 1]], 0, state["copies"])
            if pending is not None:
                results.append(pending.get())
            pending = result
        results.append(pending.get())
        return dict(state=_arrays(sim), results=np.asarray(results))
    if case["call"] == "step":
        for _ in range(case["steps"]):
            sim.Step()
        return dict(state=_arrays(sim))
    report = sim.Advance(case["steps"])
    return dict(state=_arrays(sim), report={k: float(report[k]) for k in _REPORTED})


_REPORTED = ("total_mass", "grid_mass", "kinetic_energy", "minimum_j", "maximum_j", "maximum_speed")


def work(case):
    """Each substep reads and writes the primary state once and reads the constants; a rollout's
    reverse sweep reads the states again and reads and writes their adjoints. The operations: the two
    27-node transfers, the decomposition and the return of each particle."""
    n = sum(s.particle_count for s in _scenes(case))
    dough = case["body"] != "cube"
    state = 200 if dough else (96 if case["material"] == "elastic" else 176)
    constants = 24 if dough else 8
    per_step, flops = 2 * state + constants, 3_500 if dough else 2_000
    if case["call"] == "rollout":
        per_step, flops = per_step + 3 * state + constants, 3 * flops
    return dict(bytes=float(n * case["steps"] * per_step), flops=float(n * case["steps"] * flops))


# ------------------------------------------------------------------------------------------ exact
def _det(A):
    return (A[:, 0] * torch.linalg.cross(A[:, 1], A[:, 2])).sum(1)


def _log_spd(B):
    """log of symmetric positive matrices near the identity: 2 artanh((B - I)(B + I)^-1)."""
    eye = torch.eye(3, dtype=B.dtype, device=B.device)
    Z = torch.linalg.solve(B + eye, B - eye)
    Z2 = Z @ Z
    total, power = Z, Z
    for k in range(1, 12):
        power = power @ Z2
        total = total + power / (2 * k + 1)
    return 2.0 * total


def _exp_small(A):
    eye = torch.eye(3, dtype=A.dtype, device=A.device)
    total = eye + A / 14.0
    for k in range(13, 0, -1):
        total = eye + A @ total / k
    return total


def _factor(T, knots, values):
    out = torch.full_like(T, values[0])
    for k in range(3):
        part = ((T - knots[k]) / (knots[k + 1] - knots[k])).clamp(max=1.0)
        out = torch.where(T >= knots[k], (1.0 - part) * values[k] + part * values[k + 1], out)
    return out


def _pressure_coefficient(n):
    safe = n.clamp(min=1e-300)
    return torch.where(n > 0, 9.0 / (4.0 * torch.log(1.0 / safe) ** 2 * (3.5 * n + 1.0)), torch.zeros_like(n))


def _overstress(q, p, d, h):
    """The root r of r + 1 = q / (1 + d r)^2 + p / (1 + h r)^2 (zero where q + p <= 1). Its gradient is
    that of one Newton step from the converged root."""
    def newton(r, q, p, d, h):
        u, w = 1.0 + d * r, 1.0 + h * r
        return r - (r + 1.0 - q / u ** 2 - p / w ** 2) / (1.0 + 2.0 * d * q / u ** 3 + 2.0 * h * p / w ** 3)
    with torch.no_grad():
        r = torch.zeros_like(q)
        for _ in range(40):
            new = newton(r, q, p, d, h)
            done = bool(((new - r).abs() <= 1e-15 * (1.0 + new.abs())).all())
            r = new
            if done:
                break
    return torch.where(q + p > 1.0, newton(r, q, p, d, h), torch.zeros_like(q))


def _porosity_root(q, p, d, h, e, Vp, n0):
    """The porosity n = Vp exp(e (1 - 1 / (1 + h a(n) r(n)))) - 1 + n0 of the coupled return."""
    def predicted(n):
        a = _pressure_coefficient(n)
        return Vp * torch.exp(e * (1.0 - 1.0 / (1.0 + h * a * _overstress(q, a * p, d, h * a)))) - 1.0 + n0
    n = Vp - 1.0 + n0
    with torch.enable_grad():
        for _ in range(8):
            at = n.detach().requires_grad_()
            slope, = torch.autograd.grad(predicted(at).sum(), at)
            step = (predicted(at.detach()) - at).detach() / (1.0 - slope)
            n = (at + step).detach()
            if bool((step.abs() <= 1e-15).all()):
                break
    at = n.detach()
    return at + (predicted(at) - at) / (1.0 - slope)  # the last step carries the gradient


class _Exact:
    """One body's substep in 64-bit torch; every operation differentiable."""

    def __init__(self, scene, case, s):
        self.scene, self.s0 = scene, s
        sim = scene.simulation
        self.dt, self.dx, self.R, self.bc = sim.time_step, sim.grid_spacing, sim.grid_resolution, sim.boundary_cells
        dev = s["x"].device
        self.gravity = torch.tensor(sim.gravity, dtype=torch.float64, device=dev)
        self.origin = torch.tensor(sim.grid_origin, dtype=torch.float64, device=dev)
        samples = scene.samples
        self.V = torch.as_tensor(samples.reference_volumes, device=dev)
        self.mass = torch.as_tensor(samples.particle_masses, device=dev)
        self.transport = scene.transport
        self.ding = scene.ding if scene.material.model == "ding2019" else None
        if self.transport is not None:
            t, density = scene.transport, scene.material.density
            self.dry = (density - t.water_density * t.initial_saturation) * self.V
            self.capacity = density * t.specific_heat * self.V
            mesh = scene.tet_mesh
            corners = torch.as_tensor(mesh.tet_indices, device=dev).long()[torch.as_tensor(samples.source_tets,
                                                                                           device=dev).long()]
            self.corners = corners
            vertices = torch.as_tensor(mesh.vertex_positions, device=dev)
            total = torch.zeros(len(vertices), dtype=torch.float64, device=dev)
            total.index_add_(0, corners.reshape(-1), self.V.repeat_interleave(4))
            self.corner_weight = self.V[:, None] / total[corners]
            self.corner_offset = vertices[corners] - torch.as_tensor(samples.particle_positions, device=dev)[:, None]
            faces, owners = BoundaryFaces(mesh, samples)
            self.faces = torch.as_tensor(faces, device=dev).long()
            self.owners = torch.as_tensor(owners, device=dev).long()
            self.vertex_count = len(vertices)

    # the stencil of every particle: base node, offsets, the 27 nodes (in the particles' own box) and weights
    def _stencil(self, x):
        g = (x - self.origin) / self.dx
        base = torch.floor((g - 0.5).detach()).long()
        low = base.min(0).values - 1
        self.low, shape = low, (base.max(0).values + 4 - low)
        self.shape = tuple(int(v) for v in shape)
        local = g - base
        w = [0.5 * (1.5 - local) ** 2, 0.75 - (local - 1.0) ** 2, 0.5 * (local - 0.5) ** 2]
        nodes = []
        for a in range(3):
            for b in range(3):
                for c in range(3):
                    o = torch.tensor([a, b, c], device=x.device)
                    i = base + o - low
                    flat = (i[:, 0] * self.shape[1] + i[:, 1]) * self.shape[2] + i[:, 2]
                    nodes.append((flat, w[a][:, 0] * w[b][:, 1] * w[c][:, 2], (o - local) * self.dx))
        return nodes

    def _scatter(self, nodes, values):
        """sum over particles of weight * values(d) at every node."""
        out = None
        for flat, weight, d in nodes:
            v = values(d)
            if out is None:
                out = torch.zeros(math.prod(self.shape), v.shape[1], dtype=torch.float64, device=v.device)
            out = out.index_add(0, flat, weight[:, None] * v)
        return out

    def _surface(self, s):
        t, sim = self.transport, self.scene.simulation
        n = len(s["x"])
        predicted = s["x"][:, None] + (s["F"][:, None] @ self.corner_offset[..., None])[..., 0]
        vertices = torch.zeros(self.vertex_count, 3, dtype=torch.float64, device=s["x"].device)
        vertices = vertices.index_add(0, self.corners.reshape(-1),
                                      (self.corner_weight[..., None] * predicted).reshape(-1, 3))
        p = vertices[self.faces]
        normal = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
        length = normal.norm(dim=1)
        floor = sim.grid_origin[1] + (self.bc - 1) * self.dx
        tray = (p[:, :, 1].mean(1) <= floor + t.contact_distance) & (normal[:, 1] < -0.2 * length)
        zero = torch.zeros(n, dtype=torch.float64, device=length.device)
        exposed = zero.index_add(0, self.owners, torch.where(tray, 0.0, 0.5 * length))
        contact = zero.index_add(0, self.owners, torch.where(tray, 0.5 * length, 0.0))
        saturation = s["W"] / (t.water_density * self.V * _det(s["F"]))
        loss = t.surface_water_loss * s["T"] * saturation * exposed if t.water_enabled else zero
        heat = (t.heat_transfer * exposed * (t.oven_temperature_k - s["T"])
                + t.tray_heat_transfer * contact * (t.tray_temperature_k - s["T"]) - t.latent_heat * loss)
        return heat, loss

    def _diffuse(self, f):
        """Temperature change and relative water change of every node (7-point finite volumes)."""
        t = self.transport
        vol, cap, energy, water, heat, loss = (c.reshape(self.shape) for c in f.unbind(1))
        live = cap > 0
        safe = lambda a: torch.where(live, a, torch.ones_like(a))  # noqa: E731
        T, sat = energy / safe(cap), water / (t.water_density * safe(vol))
        heat_rate, water_rate = heat, -loss
        cell = self.dx ** 3
        for axis in range(3):
            a, b = (tuple(sl if k == axis else slice(None) for k in range(3)) for sl in (slice(0, -1), slice(1, None)))
            both = live[a] & live[b]
            fill = torch.where(both, 2.0 * vol[a] * vol[b] / torch.where(both, vol[a] + vol[b], 1.0) / cell, 0.0)
            flux = t.conductivity * self.dx * fill * (T[b] - T[a])
            pad = [0, 0] * (2 - axis)
            before, after = pad + [0, 1], pad + [1, 0]
            grow = torch.nn.functional.pad
            heat_rate = heat_rate + grow(flux, before) - grow(flux, after)
            if t.water_enabled:
                flux = (t.water_diffusivity * t.water_density * self.dx * fill * 0.25 * (T[a] + T[b])
                        * (sat[a] + sat[b]) * (sat[b] - sat[a]))
                water_rate = water_rate + grow(flux, before) - grow(flux, after)
        wet = live & (water > 0)
        dT = torch.where(live, self.dt * heat_rate / safe(cap), 0.0)
        ratio = torch.where(wet, self.dt * water_rate / torch.where(wet, water, 1.0), 0.0)
        return torch.stack([dT.reshape(-1), ratio.reshape(-1)], 1)

    def _ding(self, s, C, F, T, mu, lam):
        d = self.ding
        dt, n0 = self.dt, d.porosity
        gel, T_eff = s["gelled"] != 0, T
        yield_stress, viscosity = torch.full_like(T, d.yield_stress), torch.full_like(T, d.viscosity)
        if d.temperature_enabled:
            gel = gel | (T >= d.temperature_knots_k[3])
            T_eff = torch.where(gel, d.temperature_knots_k[3], T)
            yield_stress = yield_stress * _factor(T_eff, d.temperature_knots_k, d.yield_factors)
            viscosity = viscosity * _factor(T_eff, d.temperature_knots_k, d.viscosity_factors)
        eye = torch.eye(3, dtype=torch.float64, device=T.device)
        trial = (eye + dt * C) @ s["Fe"]
        H = 0.5 * _log_spd(trial @ trial.transpose(1, 2))
        tr = H.diagonal(dim1=1, dim2=2).sum(1)
        dev = H - tr[:, None, None] / 3.0 * eye
        bulk3 = 2.0 * mu + 3.0 * lam
        mean = bulk3 * tr / 3.0
        q = 1.5 * 4.0 * mu ** 2 * (dev * dev).sum((1, 2)) / yield_stress ** 2
        p = (mean / yield_stress) ** 2
        df = 6.0 * mu * dt * yield_stress ** 2 / viscosity
        h = 2.0 / 3.0 * bulk3 * dt * yield_stress ** 2 / viscosity
        por = s["porosity"]
        if d.gas_enabled:
            por = _porosity_root(q, p, df, h, tr, 1.0 - n0 + por, n0)
        a = _pressure_coefficient(por)
        r = _overstress(q, a * p, df, a * h)
        u, w = 1.0 + df * r, 1.0 + a * h * r
        change = -dev * (1.0 - 1.0 / u)[:, None, None] - (tr / 3.0 * (1.0 - 1.0 / w))[:, None, None] * eye
        Fe = _exp_small(change) @ trial
        tau = 2.0 * mu * dev / u[:, None, None] + (mean / w)[:, None, None] * eye
        if d.gas_enabled:
            Fe = Fe * ((_det(F) / ((1.0 - n0 + por) * _det(Fe))) ** (1.0 / 3.0))[:, None, None]
        elif n0 > 0:
            por = _det(F) / _det(Fe) - 1.0 + n0
        return dict(Fe=Fe, tau=tau, porosity=por, gelled=gel.to(torch.int32))

    def step(self, s, young):
        dt, dx = self.dt, self.dx
        nu = self.scene.material.poisson_ratio
        mu, lam = young / (2.0 * (1.0 + nu)), young * nu / ((1.0 + nu) * (1.0 - 2.0 * nu))
        eye = torch.eye(3, dtype=torch.float64, device=s["x"].device)
        nodes = self._stencil(s["x"])
        new = {}
        J = _det(s["F"])
        mass, T = self.mass, s.get("T")
        if self.ding is None:
            tau = mu * (s["F"] @ s["F"].transpose(1, 2) - eye) + lam * torch.log(J)[:, None, None] * eye
        else:
            tau = s["tau"]
        if self.transport is not None:
            t = self.transport
            heat, loss = self._surface(s)
            values = torch.stack([self.V * J, self.capacity, self.capacity * s["T"], s["W"], heat, loss], 1)
            change = self._diffuse(self._scatter(nodes, lambda d: values))
            moved = sum(w[:, None] * change[flat] for flat, w, _ in nodes)
            T = s["T"] + moved[:, 0]
            new["T"], new["W"] = T, s["W"] * (1.0 + moved[:, 1])
            mass = self.dry + new["W"]
            pressure = 0.0
            if self.ding.gas_enabled:
                d = self.ding
                z = (0.5 * (s["T"] + T) - d.gas_reaction_temperature_k) / d.gas_reaction_width_k
                new["N"] = s["N"] + dt * self.scene.material.density * s["rate"] * torch.exp(-z * z)
                pressure = d.gas_ambient_pressure_pa - new["N"] * GAS_CONSTANT * T / (J * s["porosity"])
            if t.water_enabled:
                saturation = new["W"] / (t.water_density * self.V * J)
                pressure = pressure - t.water_stress * (saturation - t.initial_saturation)
            tau = tau + (J * pressure)[:, None, None] * eye
        elif self.ding is not None:
            new["T"] = T
        A = mass[:, None, None] * s["C"] - (4.0 * dt / dx ** 2 * self.V)[:, None, None] * tau
        momentum = mass[:, None] * s["v"]
        pm = self._scatter(nodes, lambda d: torch.cat([momentum + (A @ d[..., None])[..., 0], mass[:, None]], 1))
        m = pm[:, 3:]
        full = m > 0
        v = torch.where(full, pm[:, :3] / torch.where(full, m, 1.0) + dt * self.gravity, 0.0)
        index = torch.cartesian_prod(*(torch.arange(k, device=m.device) for k in self.shape)) + self.low
        walled = ((index < self.bc) & (v < 0)) | ((index >= self.R - self.bc) & (v > 0))
        v = torch.where(walled, 0.0, v)
        self.grid_mass = m.sum()
        new["v"] = sum(w[:, None] * v[flat] for flat, w, _ in nodes)
        new["C"] = 4.0 / dx ** 2 * sum((w[:, None] * v[flat])[:, :, None] * d[:, None, :] for flat, w, d in nodes)
        new["x"] = s["x"] + dt * new["v"]
        new["F"] = (eye + dt * new["C"]) @ s["F"]
        if self.ding is not None:
            new.update(self._ding(s, new["C"], new["F"], T, mu, lam))
        if "rate" in s:
            new["rate"] = s["rate"]
        return new

    def masses(self, s):
        return self.dry + s["W"] if self.transport is not None else self.mass


def _primary(s):
    """A state's outputs in the order of ``_arrays``; the gelation latch is a whole number."""
    return {k: (None if k == "gelled" else v) for k, v in s.items() if k != "rate"}


def exact(case, seed):
    if case.get("network"):
        return None  # the network is an approximation: its return has no 64-bit value
    scenes = _scenes(case)
    bodies = [(_Exact(scene, case, s), s) for k, scene in enumerate(scenes) for s in [_start(scene, case, seed, k)]]
    dev = bodies[0][1]["x"].device
    young = torch.tensor(scenes[0].material.young_modulus, dtype=torch.float64, device=dev)
    if case["call"] == "rollout":
        return _exact_rollout(case, *bodies[0], young)
    finals = []
    for body, s in bodies:
        results = []
        rate = s.get("rate")
        with torch.no_grad():
            for k in range(case["steps"]):
                if case["call"] == "graphs":
                    s = dict(s, rate=_rates(rate, k))
                s = body.step(s, young)
                results.append([body.grid_mass, (0.5 * body.masses(s) * (s["v"] ** 2).sum(1)).sum()])
        finals.append((body, s, results))
    body, s, results = finals[0]
    if case["call"] == "batch":
        sheet = [_primary(s) for _, s, _ in finals]
        return {name: None if v is None else torch.cat([b[name] for b in sheet]) for name, v in sheet[0].items()}
    if case["call"] == "graphs":
        return dict(state=_primary(s), results=np.array([[float(a), float(b)] for a, b in results]))
    if case["call"] == "step":
        return dict(state=_primary(s))
    J = _det(s["F"])
    report = dict(total_mass=body.masses(s).sum(), grid_mass=results[-1][0], kinetic_energy=results[-1][1],
                  minimum_j=J.min(), maximum_j=J.max(), maximum_speed=s["v"].norm(dim=1).max())
    return dict(state=_primary(s), report={k: float(report[k]) for k in _REPORTED})


def _exact_rollout(case, body, s, young):
    target = _target(s["x"])
    young = young.reshape(1).clone().requires_grad_()
    if body.transport is not None:
        inputs = dict(transport_temperatures="T", gas_source_rates="rate")
    else:
        inputs = dict(velocities="v")
    s = dict(s, **{k: s[k].clone().requires_grad_() for k in inputs.values()})
    leaves = dict({name: s[k] for name, k in inputs.items()}, young_modulus=young)
    for _ in range(case["steps"]):
        names = list(s)

        def step(E, *values):
            out = body.step(dict(zip(names, values)), E)
            return tuple(out[k] for k in names)

        s = dict(zip(names, checkpoint(step, young, *s.values(), use_reentrant=False)))
    loss = ((s["x"] - target) ** 2).sum(1).mean()
    gradients = torch.autograd.grad(loss, list(leaves.values()))
    names = dict(x="positions", v="velocities", C="affine_velocities", F="deformation_gradients",
                 Fe="elastic_gradients", tau="kirchhoff_stresses", porosity="porosities", N="gas_moles",
                 T="temperatures" if body.transport is None else "transport_temperatures", W="water_masses")
    state = {names[k]: v.detach() for k, v in s.items() if k in names}
    if body.transport is not None:
        state["temperatures"] = state["transport_temperatures"]  # the material's, in 32 bits
    return dict(state=state, loss=loss.detach(), gradients=dict(zip(leaves, gradients)))
