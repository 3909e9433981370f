"""P2G of bodies large enough that a block's runs are merged before they reach the grid
(csrc/bk_scatter.cuh, merge_runs): one substep of a neo-Hookean cube against the oracle.

Orders: by cell (one or two runs a warp, box of a few cells), in sample order (short runs, some kept
and some sent alone), chunks of 16 from far ends of the body in turn (kept runs too far apart for the
tile, each warp sends its own), shuffled (nothing kept). Counts: the smallest merged body and ragged
last blocks of 1 and 65 particles.

Tolerance: node sums of a few thousand float32 terms in another order, the parity bar of the grid
fields, 1e-5 of the field's norm; the summed mass within 1e-6 (a float32 rounding per node sum)."""
from dataclasses import replace

import numpy as np
import pytest

from baking_b200.config import MaterialConfig, SimulationConfig
from baking_b200.geometry import CreateDemoMesh, SampleParticles
from baking_b200.scenes import stencil_order
from tests.scenes import engine_class, set_velocity_field
from tests.test_gpu_scatter_runs import grid_of

pytestmark = pytest.mark.gpu


def build(engine, order_kind, count):
    mesh = CreateDemoMesh(2)
    per_tet = -(-count // len(mesh.tet_indices))
    s = SampleParticles(mesh, 1000., per_tet)
    keep = np.delete(np.arange(len(s.particle_positions)), np.arange(len(s.particle_positions) - count) * per_tet)
    cfg = replace(SimulationConfig(), device_name="cpu" if engine == "oracle" else "cuda:0", time_step=1e-4)
    points = s.particle_positions[keep]
    order = stencil_order(points, cfg.grid_spacing)
    if order_kind == "samples":
        order = np.arange(count)
    elif order_kind == "shuffled":
        order = np.random.default_rng(7).permutation(count)
    elif order_kind == "far":
        chunks = [order[k:k + 16] for k in range(0, count, 16)]
        half = len(chunks) // 2
        order = np.concatenate([c for pair in zip(chunks[:half], chunks[half:]) for c in pair] + chunks[2 * half:])
    at = keep[order]
    samples = replace(s, particle_positions=s.particle_positions[at], reference_volumes=s.reference_volumes[at],
                      particle_masses=s.particle_masses[at], source_tets=s.source_tets[at])
    sim = engine_class(engine)(mesh, samples, cfg, MaterialConfig())
    set_velocity_field(sim, np.array([[1.5, 0.2, 0.0], [-0.1, -0.75, 0.3], [0.0, 0.1, 0.2]], np.float32))
    return sim


@pytest.mark.parametrize("order,count", [("cells", 65536), ("cells", 65537), ("samples", 65601), ("far", 65536),
                                         ("far", 70001), ("shuffled", 65537)])
def test_merged_runs(order, count):
    ref, dev = build("oracle", order, count), build("cuda", order, count)
    assert dev.particle_data.particle_count == count
    ref.Step()
    dev.Step()
    a, b = grid_of(ref), grid_of(dev)
    for c in (slice(0, 3), slice(3, 4)):
        assert np.linalg.norm(a[:, c] - b[:, c]) <= 1e-5 * np.linalg.norm(a[:, c])
    assert abs(a[:, 3].sum() - b[:, 3].sum()) <= 1e-6 * a[:, 3].sum()
