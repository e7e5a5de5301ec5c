"""The gradient over one neighbour search per substep against the gradient that
walks the cells in every stage: the same bits."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import fluid_scene, small_mixed_scene
from test_gpu_lists import packed
from test_gpu_solver import contact_scene

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0

SCENES = {
    "one_particle": lambda bp: fluid_scene(bp, (1, 1, 1), seed=5, grid_dim=4),
    "fluid": lambda bp: fluid_scene(bp, (9, 11, 7), seed=5, grid_dim=16),
    "packed": packed,
    "contacts": lambda bp: contact_scene(bp, seed=9),
    "mixed_aliased": lambda bp: small_mixed_scene(bp, seed=29, fluid=(20, 8, 20), grid_dim=8),
    "outside": lambda bp: fluid_scene(bp, (20, 12, 16), seed=8, grid_dim=32, box=(1.0, 3.0, 1.0)),
    "large": lambda bp: fluid_scene(bp, (33, 31, 29), seed=3, grid_dim=64, box=(3.4, 4.0, 3.0)),
}


@pytest.mark.parametrize("mode", ["reference", "textbook"])
@pytest.mark.parametrize("skin,iterations", [(0.0, 3), (0.0, 1), (0.004, 2)])
@pytest.mark.parametrize("name", list(SCENES))
def test_gradients_over_the_lists_are_bit_identical_to_walks(bp, gpu, name, skin, iterations, mode):
    """Listed and (at a tiny skin) mostly queued particles, with and without
    solids and their contacts, lists past their capacity, particles that do not
    meet themselves in their walks."""
    abi = bp.abi
    m = abi.BP_MODE_TEXTBOOK if mode == "textbook" else abi.BP_MODE_REFERENCE
    scene = SCENES[name](bp)
    stages = abi.BP_STAGE_FLUID | abi.BP_STAGE_PLANES | abi.BP_STAGE_XSPH | abi.BP_STAGE_PARTICLE_COLLISION
    weights = np.random.default_rng(1).normal(size=(scene.num_particles, 3)).astype(np.float32)
    outs = []
    for walk, sk in ((abi.BP_WALK_NO_STAGING, skin), (abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS, 0.0)):
        s = bp.ParticleSolver(scene, bp.make_params(scene, mode=m, walk_options=walk, neighbor_skin=sk,
                                                    stage_mask=stages, xsph_c=0.05))
        s.tape_begin(2)
        for _ in range(2):
            s.update(2, DT, iterations)
        outs.append(s.backward(weights, 0.1 * weights))
        s.close()
    assert outs[0].keys() == outs[1].keys()
    for k in outs[0]:
        np.testing.assert_array_equal(outs[0][k], outs[1][k], err_msg=k)
