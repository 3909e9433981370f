"""A body that fits one P2G block repeats bit for bit: its node sums leave one SM in the order of the
block's warps. Finite differences of runs with nearby inputs rest on it (their quotients divide any
difference between two equal runs by the step)."""
import numpy as np
import pytest

from tests.scenes import to_np

pytestmark = pytest.mark.gpu


def test_equal_runs_of_a_small_body_are_equal():
    from tests.test_gpu_adjoint_transport import gassy_sim
    runs = []
    for _ in range(60):
        sim = gassy_sim()
        assert 128 < sim.particle_data.particle_count <= 256
        sim.AdvanceUnchecked(5)
        st = sim.current_state
        runs.append(np.concatenate([to_np(a).ravel() for a in (st.particle_positions, st.particle_velocities,
                                                               st.affine_velocities, st.deformation_gradients)]))
    for run in runs[1:]:
        np.testing.assert_array_equal(run, runs[0])
