"""Scenes of solids with the fluid stage on, whose lists hold contact partners
alone: the bits of walks without lists."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


@pytest.mark.parametrize("mode", ["reference", "textbook"])
@pytest.mark.parametrize("side,grid_dim", [(9, 16), (25, 64), (25, 8), (32, 64)])
def test_packed_solids_are_bit_identical_to_walks(bp, gpu, side, grid_dim, mode):
    """Both sides of the recording's and the readers' lines, with alias classes
    and without; contacts of every iteration from lists."""
    abi = bp.abi
    m = abi.BP_MODE_TEXTBOOK if mode == "textbook" else abi.BP_MODE_REFERENCE
    s = bp.scenes.Scene(name="grains")
    s.particle_radius, s.kernel_radius, s.cell_size, s.grid_dim = 0.05, 0.2, 0.2, grid_dim
    bp.scenes.box_planes(s, (0, 0, 0), (0.1 * side + 0.6, 9.0, 0.1 * side + 0.6))
    s.add_granulars_block((side, side, side), (0.3, 0.1, 0.3), (0.095, 0.095, 0.095), 1.0)
    s.velocities = np.random.default_rng(side).uniform(-0.5, 0.5, (s.num_particles, 3)).astype(np.float32)
    outs = []
    for walk in (abi.BP_WALK_NO_STAGING, abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS):
        g = bp.ParticleSolver(s, bp.make_params(s, mode=m, walk_options=walk))
        listed = g.walk_stats(2, DT, 3)["listed"]  # a real update
        assert (listed > 0) == (walk == abi.BP_WALK_NO_STAGING)
        for _ in range(2):
            g.update(2, DT, 3)
        outs.append((g.positions(), g.velocities(), g.field(abi.BP_FIELD_LAMBDAS)))
        g.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
