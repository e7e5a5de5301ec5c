"""Substep lists on tables of more than 2^25 cells, whose displacement bits are
shared between cells: the bits of walks without lists."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import fluid_scene, small_mixed_scene
from test_gpu_solver import contact_scene

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def wide(bp):
    """Blocks many cells apart, falling and bursting."""
    s = fluid_scene(bp, (30, 12, 14), seed=9, grid_dim=512, box=(80.0, 9.0, 60.0))
    low = s.positions.min(axis=0)
    s.positions = (low + (s.positions - low) / np.float32(1.2)).astype(np.float32)
    block = np.arange(s.num_particles) * 7 // s.num_particles  # slices of the lattice
    s.positions[:, 0] += (block * 9.7).astype(np.float32)
    s.positions[:, 2] += ((block * 3) % 7 * 7.3).astype(np.float32)
    return s


SCENES = {"wide": wide, "mixed": lambda bp: small_mixed_scene(bp, seed=5, fluid=(16, 10, 16), grid_dim=512)}


@pytest.mark.parametrize("mode", ["reference", "textbook"])
@pytest.mark.parametrize("skin", [0.0, 0.004])
@pytest.mark.parametrize("name", list(SCENES))
def test_lists_on_a_512_table_are_bit_identical_to_walks(bp, gpu, name, skin, mode):
    abi = bp.abi
    m = abi.BP_MODE_TEXTBOOK if mode == "textbook" else abi.BP_MODE_REFERENCE
    scene = SCENES[name](bp)
    outs = []
    for walk, sk in ((abi.BP_WALK_NO_STAGING, skin), (abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS, 0.0)):
        g = bp.ParticleSolver(scene, bp.make_params(scene, mode=m, walk_options=walk, neighbor_skin=sk))
        stats = g.walk_stats(2, DT, 3)  # a real update
        if sk > 0.0:
            assert stats["cells_displaced"] > 0, stats
        elif not walk & abi.BP_WALK_NO_LISTS:
            assert stats["listed"] > scene.num_particles, stats
        for _ in range(3):
            g.update(2, DT, 3)
        outs.append((g.positions(), g.velocities(), g.field(abi.BP_FIELD_DENSITIES)))
        g.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)


def test_lists_of_a_batch_with_a_512_table_are_bit_identical_to_walks(bp, gpu):
    abi = bp.abi
    scenes = [contact_scene(bp, seed=2), wide(bp), fluid_scene(bp, (8, 8, 8), seed=6, grid_dim=64)]
    outs = []
    for walk in (abi.BP_WALK_NO_STAGING, abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS):
        g = bp.BatchSolver(scenes, [bp.make_params(s, walk_options=walk, rest_density=1000.0) for s in scenes])
        for _ in range(3):
            g.step(DT, 2, 3)
        outs.append((g.positions(), g.velocities()))
        g.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)


def test_gradients_on_a_512_table_are_bit_identical_to_walks(bp, gpu):
    abi = bp.abi
    scene = wide(bp)
    stages = abi.BP_STAGE_FLUID | abi.BP_STAGE_PLANES | abi.BP_STAGE_XSPH
    weights = np.random.default_rng(1).normal(size=(scene.num_particles, 3)).astype(np.float32)
    outs = []
    for walk in (abi.BP_WALK_NO_STAGING, abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS):
        s = bp.ParticleSolver(scene, bp.make_params(scene, walk_options=walk, stage_mask=stages, xsph_c=0.05))
        s.tape_begin(2)
        s.update(2, DT, 3)
        outs.append(s.backward(weights, 0.1 * weights))
        s.close()
    for k in outs[0]:
        np.testing.assert_array_equal(outs[0][k], outs[1][k], err_msg=k)
