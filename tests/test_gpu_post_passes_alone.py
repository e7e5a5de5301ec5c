"""Post passes of a substep without a fluid stage, whose contacts alone take the
substep lists: the bits of walks without lists."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import small_mixed_scene

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


@pytest.mark.parametrize("iterations", [1, 3])
@pytest.mark.parametrize("mode,passes", [("reference", "VORTICITY"), ("reference", "VORTICITY XSPH"),
                                         ("reference", "XSPH"), ("textbook", "VORTICITY")])
def test_post_passes_beside_contact_lists_are_bit_identical_to_walks(bp, gpu, mode, passes, iterations):
    """A table much smaller than the scene: pass A's threads take class order,
    so a particle's list is in another slot than its own index.  (Textbook
    viscosity divides by the fluid stage's densities.)"""
    abi = bp.abi
    scene = small_mixed_scene(bp, seed=31, fluid=(20, 8, 20), grid_dim=8)
    stages = abi.BP_STAGE_PLANES | abi.BP_STAGE_PARTICLE_COLLISION
    for name in passes.split():
        stages |= getattr(abi, "BP_STAGE_" + name)
    m = abi.BP_MODE_TEXTBOOK if mode == "textbook" else abi.BP_MODE_REFERENCE
    outs = []
    for walk in (abi.BP_WALK_NO_STAGING, abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS):
        g = bp.ParticleSolver(scene, bp.make_params(scene, mode=m, walk_options=walk, stage_mask=stages,
                                                    vorticity_eps=0.05, xsph_c=0.1))
        stats = g.walk_stats(2, DT, iterations)  # a real update
        assert stats["alias_classes"] > 0
        if not walk & abi.BP_WALK_NO_LISTS and iterations > 1:
            assert stats["listed"] > 0
        for _ in range(2):
            g.update(2, DT, iterations)
        outs.append((g.positions(), g.velocities()))
        g.close()
    assert np.isfinite(outs[0][1]).all()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
