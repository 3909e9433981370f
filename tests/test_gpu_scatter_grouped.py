"""The scatters of bodies large enough that a warp with many runs groups its lanes by stencil base
(csrc/bk_scatter.cuh, from 256 particles on), against the oracle at ragged counts on both sides of that
line: momentum, transport fields, face owners (up to 768 particles the demo cube's owners are scattered
like particles, above it warp by warp), and the transport fields scattered ahead.

Tolerances as in test_gpu_scatter_runs.py."""
import numpy as np
import pytest

from tests.scenes import to_np
from tests.test_gpu_scatter_runs import build, grid_of

pytestmark = pytest.mark.gpu


def compare(ref, dev, T0):
    a, b = grid_of(ref), grid_of(dev)
    for c in (slice(0, 3), slice(3, 4)):
        assert np.linalg.norm(a[:, c] - b[:, c]) <= 1e-5 * np.linalg.norm(a[:, c])
    dx = ref.simulation_config.grid_spacing
    np.testing.assert_allclose(to_np(dev.current_state.particle_positions), ref.current_state.particle_positions,
                               rtol=0, atol=1e-4 * dx)
    if T0 is not None:
        change = to_np(ref.current_state.transport_state.temperatures) - T0
        got = to_np(dev.current_state.transport_state.temperatures) - T0
        assert np.abs(change).max() > 0
        assert np.linalg.norm(got - change) <= 1e-6 * np.linalg.norm(change) + 1e-13 * np.linalg.norm(T0)


@pytest.mark.parametrize("transport", [True, False])
@pytest.mark.parametrize("order", ["samples", "shuffled"])
@pytest.mark.parametrize("count", [255, 256, 257, 289, 3001])
def test_one_substep(order, count, transport):
    ref, dev = build("oracle", order, count, transport), build("cuda", order, count, transport)
    assert dev.particle_data.particle_count == count
    T0 = to_np(ref.current_state.transport_state.temperatures).copy() if transport else None
    ref.Step()
    dev.Step()
    compare(ref, dev, T0)


@pytest.mark.parametrize("count", [289, 3001])
def test_fields_scattered_ahead(count):
    ref, dev = build("oracle", "samples", count, True), build("cuda", "samples", count, True)
    T0 = to_np(ref.current_state.transport_state.temperatures).copy()
    dev.scatter_ahead = True
    dev.AdvanceUnchecked(3)
    for _ in range(3):
        ref.Step()
    compare(ref, dev, T0)
