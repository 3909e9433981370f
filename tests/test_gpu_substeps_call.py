"""Several substeps from one library call (bk_substeps) against one call per substep.

Odd and even counts (the state pair ends swapped or not), pieces that end at a periodic re-sort, both
diagnostics modes, with and without transport, and the transport fields scattered ahead. The two runs
make the same launches on the same inputs, so they differ only by the order of the grid's float
atomics: 1e-5 of each array's norm over 7 substeps (the parity bar of the grid fields)."""
import numpy as np
import pytest

from tests.scenes import baking_cube, set_velocity_field, to_np

pytestmark = pytest.mark.gpu


def one(kind, **kwargs):
    if kind == "elastic":
        from baking_b200.config import MaterialConfig, SimulationConfig
        from baking_b200.geometry import CreateDemoMesh, SampleParticles
        from baking_b200.physics.mpm import MpmSimulator
        mesh = CreateDemoMesh(2)
        sim = MpmSimulator(mesh, SampleParticles(mesh, 1000., 4), SimulationConfig(device_name="cuda:0"),
                           MaterialConfig(), **kwargs)
        rates = np.diag([1.5, -0.75, 0.2]).astype(np.float32)
    else:
        sim, rates = baking_cube("cuda")
        for name, value in kwargs.items():
            setattr(sim, name, value)
    set_velocity_field(sim, rates)
    return sim


def arrays_of(sim):
    st = sim.current_state
    out = [st.particle_positions, st.particle_velocities, st.deformation_gradients]
    if st.material_state is not None:
        out += [st.material_state.elastic_gradients, st.material_state.plastic_gradients]
    if st.transport_state is not None:
        t = st.transport_state
        out += [t.temperatures, t.water_masses, t.water_losses, t.heat_exchanges]
    order = np.argsort(sim.particle_order.cpu().numpy())  # back to the constructor's particle order
    return [to_np(a).astype(np.float64)[order] for a in out]


@pytest.mark.parametrize("kind,count,kwargs,ahead", [
    ("dough", 7, {}, False), ("dough", 4, dict(diagnostics="lean"), False), ("dough", 7, dict(sort_interval=3), False),
    ("dough", 6, {}, True), ("dough", 1, {}, False), ("elastic", 5, {}, False),
    ("elastic", 6, dict(sort_interval=2), False)])
def test_many_substeps_match_single_substeps(kind, count, kwargs, ahead):
    a, b = one(kind, **kwargs), one(kind, **kwargs)
    a.scatter_ahead = ahead
    a.AdvanceUnchecked(count)
    for _ in range(count):
        b._substep(check=False)
    assert a.step_count == b.step_count == count and a.sort_count == b.sort_count
    assert (a._current is not None) and (a._engine.prescatter_pending is False)
    for x, y in zip(arrays_of(a), arrays_of(b)):
        assert np.isfinite(x).all()
        assert np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(y) + 1e-30
    report = a.CheckState()
    assert report["step_count"] == count
    # the simulator goes on from there
    a.AdvanceUnchecked(1)
    b.AdvanceUnchecked(1)
    for x, y in zip(arrays_of(a), arrays_of(b)):
        assert np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(y) + 1e-30
