"""Conduction inside an insulated body conserves its energy: the scalar P2G and G2P use the same weights, so
what a node loses arrives at others to the last float64 place.

Bound: every substep rounds every temperature once (2^-53 of it, random signs), four standard deviations
of the sum over the body, relative to the heat that moved."""
from dataclasses import replace

import numpy as np
import pytest

from tests.scenes import to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("voxels,per_tet", [(2, 4), (4, 5), (11, 5)])
def test_energy_of_an_insulated_body(voxels, per_tet):
    import torch
    from baking_b200.config import DingConfig, MaterialConfig, SimulationConfig, TransportConfig
    from baking_b200.geometry import CreateDemoMesh, SampleParticles
    from baking_b200.physics.mpm import MpmSimulator
    mesh, steps = CreateDemoMesh(voxels), 100
    sim = MpmSimulator(
        mesh, SampleParticles(mesh, 1000., per_tet),
        replace(SimulationConfig(), device_name="cuda:0", time_step=1e-4, gravity=(0., 0., 0.)),
        MaterialConfig(model="ding2019", young_modulus=2e4), ding_config=DingConfig(porosity=0.1),
        transport_config=TransportConfig(enabled=True, initial_temperature_k=330.0, conductivity=20.,
                                         specific_heat=100., heat_transfer=0., tray_heat_transfer=0.,
                                         water_enabled=False), diagnostics="lean")
    x = to_np(sim.current_state.particle_positions).astype(np.float64)
    T = 330 + 20 * np.sin(25 * x[:, 0] + 3) * np.cos(31 * x[:, 1]) + 5 * np.random.default_rng(0).standard_normal(len(x))
    sim.current_state.transport_state.temperatures.copy_(torch.as_tensor(T, device="cuda"))
    capacity = to_np(sim.transport.capacities).astype(np.longdouble)
    sim.AdvanceUnchecked(steps)
    after = to_np(sim.current_state.transport_state.temperatures)
    moved = float((capacity * np.abs(after - T)).sum())
    drift = float((capacity * after).sum() - (capacity * T).sum())
    assert moved > 1e-5 * float((capacity * T).sum())
    assert abs(drift) <= 4 * 2.0 ** -53 * 330 * np.sqrt(steps * float((capacity ** 2).sum()))
