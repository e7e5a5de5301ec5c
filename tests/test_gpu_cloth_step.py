"""The one-launch end of a cloth iteration (distance constraints, immovables,
planes or commit) against the launches it replaces: the same bits."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import fluid_scene

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def cloth(bp, n, pinned=True, fluid=False):
    s = fluid_scene(bp, (4, 3, 4), seed=8, grid_dim=16) if fluid else bp.scenes.flag_scene(n=n, floor=0.5)
    if fluid:
        s.add_cloth((0.1, 0.45, 0.1), (0.1, 0, 0), (0, 0, 0.1), n, n, 1.0, stretch=0.25, shear=0.1, bend=0.05)
    s.add_rope((0.3, 1.6, 0.2), (0.3, 0.9, 0.2), 6, 0.5)
    # a doubled edge, one of no length and one from a particle to itself
    extra = np.array([[0, 1], [0, 1], [2, 2]], np.int32) + (s.num_particles - 6)
    s._add_pairs(extra, np.array([[0.1, 0.5], [0.2, 0.1], [0.1, 0.5]], np.float32))
    if not pinned:
        s.immovables = np.zeros(0, np.int32)
    rng = np.random.default_rng(4)
    s.velocities = rng.uniform(-0.5, 0.5, (s.num_particles, 3)).astype(np.float32)
    return s


@pytest.mark.parametrize("iterations", [1, 4])
@pytest.mark.parametrize("n,pinned,fluid", [(2, True, False), (3, False, False), (11, True, False), (33, True, False),
                                            (8, True, True), (8, False, True)])
def test_cloth_step_is_bit_identical(bp, gpu, n, pinned, fluid, iterations):
    abi = bp.abi
    scene = cloth(bp, n, pinned, fluid)
    outs = []
    for walk in (abi.BP_WALK_NO_STAGING, abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_FUSION):
        g = bp.ParticleSolver(scene, bp.make_params(scene, walk_options=walk, mass_scaling_k=0.0))
        for _ in range(4):
            g.update(2, DT, iterations)
        outs.append((g.positions(), g.velocities(), g.field(abi.BP_FIELD_NEW_POSITIONS), g.last_launch_count()))
        g.close()
    assert outs[0][3] < outs[1][3]  # fewer launches
    for a, b in zip(outs[0][:3], outs[1][:3]):
        np.testing.assert_array_equal(a, b)
