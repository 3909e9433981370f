"""Surface vertices of coarse meshes come out bit for bit the same from the launch they share with the
transport scatter and from their own (which substeps on fields scattered ahead take, and whose form
the reverse sweep recomputes them with): meshes of 123, 264 and 1,325 bindings a
vertex (a warp, 128 and 256 threads each)."""
import numpy as np
import pytest

from tests.scenes import to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("resolution,particles,low,high", [(64, 28_001, 1, 127), (64, 60_001, 128, 1023),
                                                           (64, 300_001, 1024, 10_000)])
def test_shared_and_own_launch(resolution, particles, low, high):
    import torch
    from baking_b200.physics.substep import PHASE_TRANSPORT
    from baking_b200.scenes import box_loaf, make_simulator
    sim = make_simulator(box_loaf(resolution, particles, 0), diagnostics="lean")
    g = torch.Generator(device="cuda").manual_seed(1)  # every binding predicts another position
    F = sim.current_state.deformation_gradients
    F += 0.02 * torch.randn(F.shape, generator=g, device="cuda")
    eng = sim._engine
    assert eng.surface.vertex_count > 0 and eng.surface.owner_count * 16 < sim.particle_data.particle_count
    assert low <= eng.surface_bindings // eng.surface.vertex_count <= high
    vertices = sim.surface_vertices_buffer()
    out = []
    for ahead in (False, True):
        vertices.zero_()
        eng.prescatter_pending = ahead
        eng.run(sim._current, sim.next_state, False, PHASE_TRANSPORT, False, prescattered=ahead)
        out.append(to_np(vertices).copy())
    assert np.abs(out[0]).max() > 0
    np.testing.assert_array_equal(out[1], out[0])
