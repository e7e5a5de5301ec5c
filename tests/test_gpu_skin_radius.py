"""The adapted skin of the substep lists where the kernel radius changes on a
live solver."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import fluid_scene

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def test_skin_follows_a_smaller_radius(bp, gpu):
    """A lattice of spacing h / 2 for a radius h set after creation, a twentieth
    of the radius before: the lists serve as many reads as those of a solver
    created with h (a skin kept as a length would overflow them)."""
    abi = bp.abi
    scene = fluid_scene(bp, (20, 20, 20), seed=3, grid_dim=16)
    low = scene.positions.min(axis=0)
    scene.positions = (np.float32(1.0) + (scene.positions - low) * np.float32(0.05)).astype(np.float32)
    scene.velocities[:] = 0.0
    scene.masses[:] = 1000.0 * 0.005 ** 3
    over = dict(mode=abi.BP_MODE_TEXTBOOK, walk_options=abi.BP_WALK_NO_STAGING)
    small = bp.make_params(scene, kernel_radius=0.01, **over)
    g = bp.ParticleSolver(scene, bp.make_params(scene, **over))
    g.set_params(small)
    fresh = bp.ParticleSolver(scene, small)
    want = fresh.walk_stats(1, DT / 2, 4)  # real updates
    assert want["listed"] > 2 * scene.num_particles
    assert g.walk_stats(1, DT / 2, 4) == want
    np.testing.assert_array_equal(g.positions(), fresh.positions())
    g.close()
    fresh.close()


@pytest.mark.parametrize("mode", ["reference", "textbook"])
@pytest.mark.parametrize("grid_dim", [4, 32])
def test_lists_after_radius_changes_are_bit_identical_to_walks(bp, gpu, grid_dim, mode):
    """Radii lowered and raised between updates, on a table much smaller than
    the scene and on a roomy one: the bits of walks without lists."""
    abi = bp.abi
    m = abi.BP_MODE_TEXTBOOK if mode == "textbook" else abi.BP_MODE_REFERENCE
    scene = fluid_scene(bp, (14, 12, 15), seed=12, grid_dim=grid_dim)
    outs = []
    for walk in (abi.BP_WALK_NO_STAGING, abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS):
        g = bp.ParticleSolver(scene, bp.make_params(scene, mode=m, walk_options=walk))
        out = []
        for radius in (0.2, 0.13, 0.18, 0.11):
            g.set_params(bp.make_params(scene, mode=m, walk_options=walk, kernel_radius=radius))
            for _ in range(2):
                g.update(2, DT, 3)
            out += [g.positions(), g.velocities()]
        outs.append(out)
        g.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
