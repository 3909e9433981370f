"""How a run of unchecked substeps is cut into library calls, on the CPU: a stand-in engine notes the calls
and steps a number instead of a state."""
import numpy as np
import pytest

from baking_b200.physics.mpm import MpmSimulator


class Engine:
    def __init__(self, fail_at=None):
        self.calls, self.done, self.fail_at = [], 0, fail_at

    def prescatter_allowed(self):
        return False

    def run_many(self, state, other, count, full, ahead):
        self.calls.append(count)
        pair = [state, other]
        for k in range(count):
            if self.done == self.fail_at:
                error = RuntimeError("launch failed")
                error.launched = k
                raise error
            pair[1 - k % 2]["steps"] = pair[k % 2]["steps"] + 1
            self.done += 1


def simulator(sort_interval=0, fail_at=None):
    sim = MpmSimulator.__new__(MpmSimulator)
    sim.transport, sim.retain_history, sim.diagnostics, sim.scatter_ahead = None, False, "lean", False
    sim.sort_interval, sim.step_count, sim._stale, sim._baking_start_step = sort_interval, 0, False, 0
    sim._current, sim.next_state = dict(steps=0), dict(steps=0)
    sim._engine = Engine(fail_at)
    sim.sorts = []
    sim.SortParticles = lambda: sim.sorts.append(sim.step_count)
    return sim


@pytest.mark.parametrize("count", [0, 1, 2, 63, 64, 65, 130])
@pytest.mark.parametrize("sort_interval", [0, 7, 100])
def test_pieces(count, sort_interval):
    sim = simulator(sort_interval)
    sim.AdvanceUnchecked(np.int64(count))
    assert sim.step_count == sim._current["steps"] == sum(sim._engine.calls) == count
    assert max(sim._engine.calls, default=0) <= 64  # an interrupt waits for no more than that
    assert sim._stale == (count > 0)
    assert sim.sorts == [k for k in range(1, count + 1) if sort_interval and k % sort_interval == 0]


@pytest.mark.parametrize("fail_at", [0, 1, 2, 63, 64, 67, 128])
def test_a_failing_launch_leaves_the_last_complete_substep(fail_at):
    sim = simulator(fail_at=fail_at)
    with pytest.raises(RuntimeError, match="launch failed"):
        sim.AdvanceUnchecked(130)
    assert sim.step_count == sim._current["steps"] == fail_at
    assert sim._stale == (fail_at > 0)


@pytest.mark.parametrize("count", [2.5, 2.0, "2", None, np.float32(3)])
def test_counts_that_are_no_whole_numbers_are_refused(count):
    sim = simulator()
    for call in (sim.AdvanceUnchecked, sim.Advance):
        with pytest.raises(TypeError):
            call(count)
    assert sim.step_count == 0 and not sim._engine.calls
