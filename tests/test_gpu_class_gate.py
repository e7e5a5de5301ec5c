"""Alias classes that close inside a substep, after its lists were recorded:
the bits of walks without classes."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import fluid_scene

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


@pytest.mark.parametrize("mode", ["reference", "textbook"])
@pytest.mark.parametrize("fluid", [(20, 6, 20), (28, 40, 28)])
def test_classes_closing_after_the_recording_leave_the_bits(bp, gpu, fluid, mode):
    """An edge compressed from a length of 3 throws its ends further than the
    reach in the first iteration's constraint stage, behind the pass that
    recorded the lists; a rope lies on the fluid, whose later passes gather
    its particles.  Sizes of the four-lane and of the one-thread readers.
    (Without Akinci tension reference densities below rest are not clamped.)"""
    abi = bp.abi
    m = abi.BP_MODE_TEXTBOOK if mode == "textbook" else abi.BP_MODE_REFERENCE
    top = 0.1 * fluid[1]
    scene = fluid_scene(bp, fluid, seed=17, grid_dim=8, box=(3.0, top + 4.0, 3.0))
    scene.add_rope((0.3, top + 0.07, 0.3), (1.7, top + 0.07, 1.6), 15, 1.0)
    scene.add_rope((0.5, top + 2.0, 0.5), (0.7, top + 2.0, 0.5), 2, 1.0)
    scene.distance_params[-1] = (3.0, 1.0)
    outs = []
    for walk in (abi.BP_WALK_NO_STAGING, abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_ALIAS_CLASSES):
        g = bp.ParticleSolver(scene, bp.make_params(scene, mode=m, walk_options=walk, mass_scaling_k=0.0,
                                                    stage_mask=abi.BP_STAGE_ALL & ~abi.BP_STAGE_AKINCI))
        stats = g.walk_stats(1, DT / 2, 3)  # a real update
        if not walk & abi.BP_WALK_NO_ALIAS_CLASSES:
            n = scene.num_particles
            assert 0 < stats["alias_classes"] < 1.5 * n, stats  # the recording alone took them
            assert stats["cells_no_list"] > 2 * n  # every later reader found the slots changed
        for _ in range(2):
            g.update(1, DT / 2, 3)
        outs.append((g.positions(), g.velocities(), g.field(abi.BP_FIELD_DENSITIES), g.field(abi.BP_FIELD_LAMBDAS)))
        g.close()
    assert np.isfinite(outs[1][1]).all()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
