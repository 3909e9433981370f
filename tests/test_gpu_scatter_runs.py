"""The particle-to-grid scatters (csrc/bk_scatter.cuh) over the particle orders that shape a warp's runs.

One checked substep of the demo cube (Ding, gas, thermal-water transport; and neo-Hookean without
transport) against the oracle, with the particles by cell (long contiguous runs), in sample order
(tet by tet: many short runs, grouped within the warp), shuffled (nearly every lane a base of its
own) and cut to ragged counts (a last warp of 1, 31 or 33 particles, a lone particle).

Tolerances. Node sums of up to a few hundred float32 terms in another order: the parity bar of the
grid fields, 1e-5 of the field's norm. Temperatures: the node changes dT are float64 sums weighted
by float32 products, equal to 1e-6 of the change itself."""
from dataclasses import replace

import numpy as np
import pytest

from baking_b200.config import DingConfig, MaterialConfig, SimulationConfig, TransportConfig
from baking_b200.geometry import CreateDemoMesh, SampleParticles
from baking_b200.scenes import stencil_order
from tests.scenes import engine_class, set_velocity_field, to_np

pytestmark = pytest.mark.gpu


def build(engine, order_kind, keep, transport):
    mesh = CreateDemoMesh(2 if keep > 40 else 1)
    # every tet needs a particle: ragged counts come from the last tets' extra samples
    per_tet = max(1, -(-keep // len(mesh.tet_indices)))
    s = SampleParticles(mesh, 1000., per_tet)
    n = len(s.particle_positions)
    drop = np.zeros(n, dtype=bool)
    drop[[t * per_tet + k for k in range(per_tet - 1) for t in range(len(mesh.tet_indices))][:n - keep]] = True
    keep_at = np.flatnonzero(~drop)
    cfg = replace(SimulationConfig(), device_name="cpu" if engine == "oracle" else "cuda:0", time_step=1e-4)
    points = s.particle_positions[keep_at]
    order = {"cells": stencil_order(points, cfg.grid_spacing), "samples": np.arange(len(points)),
             "shuffled": np.random.default_rng(7).permutation(len(points))}[order_kind]
    at = keep_at[order]
    samples = replace(s, particle_positions=s.particle_positions[at], reference_volumes=s.reference_volumes[at],
                      particle_masses=s.particle_masses[at], source_tets=s.source_tets[at])
    if transport:
        sim = engine_class(engine)(
            mesh, samples, cfg, MaterialConfig(model="ding2019", young_modulus=2e4),
            ding_config=DingConfig(gas_enabled=True, porosity=0.2, yield_stress=200., viscosity=1e6,
                                   temperature_enabled=True, gas_production_rate=0.01),
            transport_config=TransportConfig(enabled=True, initial_temperature_k=330.0, heat_transfer=2000.,
                                             conductivity=20., specific_heat=100., water_diffusivity=1e-8,
                                             surface_water_loss=1e-5))
    else:
        sim = engine_class(engine)(mesh, samples, cfg, MaterialConfig())
    rates = np.array([[1.5, 0.2, 0.0], [-0.1, -0.75, 0.3], [0.0, 0.1, 0.2]], np.float32)
    set_velocity_field(sim, rates)
    return sim


def grid_of(sim):
    if hasattr(sim, "grid_masses"):
        return np.concatenate([sim.grid_momenta, sim.grid_masses[:, None]], axis=1).astype(np.float64)
    return to_np(sim.grid_state.node_pm).astype(np.float64)


@pytest.mark.parametrize("transport", [True, False])
@pytest.mark.parametrize("order,count", [("cells", 192), ("samples", 192), ("shuffled", 192), ("samples", 191),
                                         ("shuffled", 65), ("cells", 63), ("samples", 24), ("cells", 6)])
def test_one_substep_in_any_particle_order(order, count, transport):
    ref, dev = build("oracle", order, count, transport), build("cuda", order, count, transport)
    assert dev.particle_data.particle_count == count
    T0 = to_np(ref.current_state.transport_state.temperatures).copy() if transport else None
    ref.Step()
    dev.Step()
    a, b = grid_of(ref), grid_of(dev)
    for c in (slice(0, 3), slice(3, 4)):
        assert np.linalg.norm(a[:, c] - b[:, c]) <= 1e-5 * np.linalg.norm(a[:, c])
    dx = ref.simulation_config.grid_spacing
    np.testing.assert_allclose(to_np(dev.current_state.particle_positions), ref.current_state.particle_positions,
                               rtol=0, atol=1e-4 * dx)
    if transport:
        change = to_np(ref.current_state.transport_state.temperatures) - T0
        got = to_np(dev.current_state.transport_state.temperatures) - T0
        assert np.abs(change).max() > 0
        assert np.linalg.norm(got - change) <= 1e-6 * np.linalg.norm(change) + 1e-13 * np.linalg.norm(T0)
