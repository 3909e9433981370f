"""The node box of a substep whose phases or scatters come from different calls.

P2G relies on the box that the transport scatter of the same call widened, and has to widen it itself in
every other case: checked substeps (two calls each) on transport fields scattered ahead, as Advance
makes them while a body settles, and mechanics phases alone with transport on, through bk_substep and
through an instance table.

The compared runs make the same substeps on the same values, so they differ by the order of the
grid's float atomics: 1e-5 of each array's norm (the parity bar of the grid fields)."""
from dataclasses import replace

import numpy as np
import pytest

from tests.scenes import baking_cube, build_gas, set_velocity_field, to_np

pytestmark = pytest.mark.gpu

DT = 1e-4


def arrays_of(sim):
    st = sim.current_state
    out = dict(x=st.particle_positions, v=st.particle_velocities, C=st.affine_velocities, F=st.deformation_gradients,
               pm=sim.grid_state.node_pm)
    if st.transport_state is not None:
        out.update(T=st.transport_state.temperatures, W=st.transport_state.water_masses)
    return {k: to_np(v).astype(np.float64) for k, v in out.items()}


def compare(a, b):
    a, b = arrays_of(a), arrays_of(b)
    assert np.linalg.norm(b["v"]) > 0 and np.linalg.norm(b["C"]) > 0
    for name in b:
        assert np.linalg.norm(a[name] - b[name]) <= 1e-5 * np.linalg.norm(b[name]), name


def settling(steps):
    sim, rates = baking_cube("cuda")
    config = replace(sim.transport.config, settling_duration_s=steps * DT)
    sim = type(sim)(sim.tet_mesh, sim.particle_samples, sim.simulation_config, sim.material.material_config,
                    ding_config=sim.material.ding_config, transport_config=config)
    set_velocity_field(sim, rates)
    return sim


@pytest.mark.parametrize("settle,advance", [(1000, 4), (3, 6), (1, 2), (2, 3)])
def test_settling_with_the_scatter_ahead(settle, advance):
    a, b = settling(settle), settling(settle)
    a.scatter_ahead = True
    assert a.IsSettling
    a.Advance(advance)
    for _ in range(advance):
        b.Step()
    assert a.IsSettling == b.IsSettling == (settle > advance)
    compare(a, b)
    a.Advance(2)  # on a grid that has to be clean behind it
    b.Step()
    b.Step()
    compare(a, b)


def still_transport():
    """A body whose transport changes nothing: no conduction, no heat or water exchange."""
    sim = build_gas("cuda")
    set_velocity_field(sim, np.array([[1.5, 0.2, 0.0], [-0.1, -0.75, 0.3], [0.0, 0.1, 0.2]], np.float32))
    return sim


@pytest.mark.parametrize("table", [False, True])
def test_mechanics_alone_on_a_fresh_grid(table):
    from baking_b200 import _lib
    from baking_b200.batch import BatchedSimulators
    from baking_b200.physics.substep import PHASE_MECHANICS
    a, b = still_transport(), still_transport()
    batch = BatchedSimulators([a], launch="table") if table else None
    if table:
        batch._ensure_layout()
    for k in range(4):
        if table:
            _lib.call_raw(a._engine.lib.bk_batch_substep, "bk_batch_substep", batch._tables[0], k % 2, PHASE_MECHANICS,
                          0, 0, _lib.stream_handle())
        else:
            a._engine.run(a._current, a.next_state, False, PHASE_MECHANICS, False)
        a._current, a.next_state = a.next_state, a._current
        b.Step()
    a._stale = True
    compare(a, b)


@pytest.mark.parametrize("subdivisions", [1, 3])
def test_passes_over_a_sparse_box(subdivisions):
    """Two halves of a small cube in far corners: the node box holds thousands of nodes for every
    particle, and its passes are shared by enough blocks that a substep stays within 8 times that
    of the compact cube (the box passes move some 100 MB: two substeps' time; with blocks counted by
    particles it took 30 times)."""
    import torch
    times = []
    for apart in (0.0, 0.25):
        sim, _ = baking_cube("cuda", subdivisions=subdivisions, gravity=(0., 0., 0.), dt=1e-6)
        sim = type(sim)(sim.tet_mesh, sim.particle_samples, replace(sim.simulation_config, grid_resolution=128,
                                                                    grid_spacing=1.0 / 128),
                        sim.material.material_config, ding_config=sim.material.ding_config,
                        transport_config=sim.transport.config, diagnostics="lean")
        x, half = sim.current_state.particle_positions, sim.particle_data.particle_count // 2
        x[:half] += apart
        x[half:] -= apart
        best = float("inf")
        for _ in range(4):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            sim.AdvanceUnchecked(20)
            end.record()
            torch.cuda.synchronize()
            best = min(best, start.elapsed_time(end))
        times.append(best)
    assert times[1] <= 8.0 * times[0], times
