"""Walk mode: textbook scenes past the four-lane readers whose substep lists would
not pay walk in every pass instead, and go back to lists; the bits of walks
without lists throughout."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import fluid_scene

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def squeezed(bp, n, grid_dim, cloth=0):
    """Fluid at 1 / 1.3 of its rest spacing, where corrections move most
    particles past the skin; a cloth just above it."""
    scene = fluid_scene(bp, n, seed=n[0], grid_dim=grid_dim, box=(8.0, 8.0, 8.0))
    low = scene.positions.min(axis=0)
    scene.positions = (low + (scene.positions - low) / np.float32(1.3)).astype(np.float32)
    if cloth:
        top = float(scene.positions[:, 1].max())
        scene.add_cloth((0.5, top + 0.08, 0.5), (0.1, 0, 0), (0, 0, 0.1), cloth, cloth, 1.0)
    return scene


CASES = {
    # the walks' planes: from the position pass, with the class refresh, none, in launches of their own
    "fluid": (lambda bp: squeezed(bp, (40, 36, 34), 128), "POST"),
    "aliased": (lambda bp: squeezed(bp, (40, 36, 34), 16), "POST"),
    "cloth": (lambda bp: squeezed(bp, (40, 36, 34), 128, cloth=16), "POST"),
    "large": (lambda bp: squeezed(bp, (64, 56, 60), 128, cloth=16), "POST"),
    "viscosity": (lambda bp: squeezed(bp, (40, 36, 34), 128), "XSPH"),
    "viscosity_aliased": (lambda bp: squeezed(bp, (40, 36, 34), 16), "XSPH"),
}


def params(bp, scene, walk, post):
    abi = bp.abi
    stages = abi.BP_STAGE_ALL if post == "POST" else abi.BP_STAGE_ALL & ~(abi.BP_STAGE_VORTICITY | abi.BP_STAGE_AKINCI)
    return bp.make_params(scene, mode=abi.BP_MODE_TEXTBOOK, walk_options=walk, stage_mask=stages, xsph_c=0.05,
                          mass_scaling_k=0.0)


@pytest.mark.parametrize("name", list(CASES))
def test_walk_mode_is_bit_identical_to_walks(bp, gpu, name):
    """A squeezed block set back again and again, then one at rest: lists at
    first, walks while it bursts, lists at rest."""
    abi = bp.abi
    make, post = CASES[name]
    scene = make(bp)
    n = scene.num_particles
    rest = scene.positions.copy()
    fluid = scene.phases < 0
    low = rest[fluid].min(axis=0)
    rest[fluid] = low + (rest[fluid] - low) * np.float32(1.3)
    rest[~fluid, 1] += np.float32(3.0)
    a, b = (bp.ParticleSolver(scene, params(bp, scene, w, post))
            for w in (abi.BP_WALK_NO_STAGING, abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS))
    listed = []
    for k in range(32):  # 20 updates at rest: the last of 8 substeps lets the skin shrink by a third
        if k % 2 == 0:
            for s in (a, b):
                s.set_state(scene.positions if k < 12 else rest, np.zeros((n, 3), np.float32))
        listed.append(a.walk_stats(2, DT, 4)["listed"])  # a real update
        b.update(2, DT, 4)
        np.testing.assert_array_equal(a.positions(), b.positions())
        np.testing.assert_array_equal(a.velocities(), b.velocities())
    a.close()
    b.close()
    # contacts read their lists in any mode: few particles near the cloth
    assert min(listed[2:12]) < n // 2, listed
    assert max(listed[12:]) > 2 * n, listed


def test_gradients_in_walk_mode_are_bit_identical_to_walks(bp, gpu):
    """A recording whose substeps, and whose re-run, walk."""
    abi = bp.abi
    scene = squeezed(bp, (40, 36, 34), 128)
    weights = np.random.default_rng(1).normal(size=(scene.num_particles, 3)).astype(np.float32)
    outs = []
    for walk in (abi.BP_WALK_NO_STAGING, abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS):
        s = bp.ParticleSolver(scene, params(bp, scene, walk, "XSPH"))
        for _ in range(6):
            s.set_state(scene.positions, np.zeros_like(scene.positions))
            stats = s.walk_stats(2, DT, 4)
        assert stats["listed"] == 0, stats
        s.set_state(scene.positions, np.zeros_like(scene.positions))
        s.tape_begin(4)
        s.update(2, DT, 3)
        outs.append(dict(s.backward(weights, 0.1 * weights), x=s.positions()))
        s.close()
    for k in outs[0]:
        np.testing.assert_array_equal(outs[0][k], outs[1][k], err_msg=k)
