"""The substep lists (one neighbour search per substep) against walks of the
cells: the same bits, where lists are read and where particles must walk."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import fluid_scene, small_mixed_scene
from test_gpu_solver import contact_scene

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def grains(bp, grid_dim=16):
    """Grains alone (no fluid): the lists hold contact partners only."""
    s = bp.scenes.Scene(name="grains")
    s.particle_radius, s.kernel_radius, s.cell_size, s.grid_dim = 0.05, 0.2, 0.2, grid_dim
    bp.scenes.box_planes(s, (0, 0, 0), (1.6, 3.0, 1.6))
    s.add_granulars_block((7, 6, 7), (0.3, 0.2, 0.3), (0.09, 0.09, 0.09), 1.0)
    rng = np.random.default_rng(3)
    s.velocities = rng.uniform(-1.0, 1.0, (s.num_particles, 3)).astype(np.float32)
    return s


def packed(bp):
    """A core at 0.4 of the spacing: its lists overflow (about 500 neighbours
    within h), and those around it hold up to their capacity."""
    s = fluid_scene(bp, (12, 12, 12), seed=41, grid_dim=16)
    x = s.positions.copy()
    c = x.mean(axis=0)
    core = np.all(np.abs(x - c) < 0.35, axis=1)
    x[core] = c + (x[core] - c) * np.float32(0.4)
    s.positions = x.astype(np.float32)
    return s


SCENES = {
    "fluid": lambda bp: fluid_scene(bp, (9, 11, 7), seed=5, grid_dim=16),
    "one_particle": lambda bp: fluid_scene(bp, (1, 1, 1), seed=5, grid_dim=4),
    "packed": packed,
    "contacts": lambda bp: contact_scene(bp, seed=9),
    "grains": grains,
    "grains_aliased": lambda bp: grains(bp, grid_dim=4),
    "mixed_aliased": lambda bp: small_mixed_scene(bp, seed=29, fluid=(20, 8, 20), grid_dim=8),
}


@pytest.mark.parametrize("mode", ["reference", "textbook"])
@pytest.mark.parametrize("skin,iterations", [(0.0, 4), (0.0, 1), (0.1, 2), (0.004, 5)])
@pytest.mark.parametrize("name", list(SCENES))
def test_substep_lists_are_bit_identical_to_walks(bp, gpu, name, skin, iterations, mode):
    """Adapted and fixed skins (one so small that most particles are queued),
    an odd and an even number of list passes, and a substep whose only readers
    are the post passes: the bits of walks without lists."""
    abi = bp.abi
    m = abi.BP_MODE_TEXTBOOK if mode == "textbook" else abi.BP_MODE_REFERENCE
    scene = SCENES[name](bp)
    outs = []
    for walk, sk in ((abi.BP_WALK_NO_STAGING, skin), (abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS, 0.0)):
        g = bp.ParticleSolver(scene, bp.make_params(scene, mode=m, walk_options=walk, neighbor_skin=sk))
        listed = g.walk_stats(2, DT, iterations)["listed"]  # a real update
        if walk & abi.BP_WALK_NO_LISTS:
            assert listed == 0
        elif sk != 0.004 and (iterations > 1 or not name.startswith("grains")):
            assert listed > 0
        for _ in range(3):
            g.update(2, DT, iterations)
        outs.append((g.positions(), g.velocities(), g.field(abi.BP_FIELD_DENSITIES), g.field(abi.BP_FIELD_LAMBDAS)))
        g.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)


def test_substep_lists_in_a_batch_with_solids(bp, gpu):
    """Scenes of different grids and phases in one solver: lists against walks."""
    abi = bp.abi
    scenes = [contact_scene(bp, seed=2), fluid_scene(bp, (8, 8, 8), seed=6, grid_dim=32), grains(bp)]
    outs = []
    for walk in (abi.BP_WALK_NO_STAGING, abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS):
        g = bp.BatchSolver(scenes, [bp.make_params(s, walk_options=walk, rest_density=1000.0) for s in scenes])
        for _ in range(4):
            g.step(DT, 2, 3)
        outs.append((g.positions(), g.velocities()))
        g.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("mode", ["reference", "textbook"])
@pytest.mark.parametrize("side", [24, 31, 36])
def test_readers_and_recorders_by_size(bp, gpu, side, mode):
    """Scenes around the sizes where the recording launch takes a warp or a
    thread per particle and the readers four lanes or one: lists against
    walks, with a cloth's contacts and lists of every length at the walls."""
    abi = bp.abi
    m = abi.BP_MODE_TEXTBOOK if mode == "textbook" else abi.BP_MODE_REFERENCE
    scene = fluid_scene(bp, (side, side, side), seed=side, grid_dim=64, box=(4.0, 4.0, 4.0))
    scene.add_cloth((0.5, 0.1 * side + 0.15, 0.5), (0.1, 0, 0), (0, 0, 0.1), 9, 9, 1.0)
    scene.velocities[-81:, 1] = -2.0
    outs = []
    for walk in (abi.BP_WALK_NO_STAGING, abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS):
        g = bp.ParticleSolver(scene, bp.make_params(scene, mode=m, walk_options=walk))
        for _ in range(3):
            g.update(2, DT, 3)
        outs.append((g.positions(), g.velocities(), g.field(abi.BP_FIELD_DENSITIES), g.field(abi.BP_FIELD_LAMBDAS)))
        g.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("mode", ["reference", "textbook"])
@pytest.mark.parametrize("grid_dim", [16, 64])
@pytest.mark.parametrize("n", [(20, 12, 16), (40, 36, 20), (40, 36, 34)])
def test_lists_of_particles_far_from_their_stored_cells(bp, gpu, n, grid_dim, mode):
    """A block partly outside its box: the planes move particles cells away from
    the ones they are stored in, so that their walks do not meet themselves."""
    abi = bp.abi
    m = abi.BP_MODE_TEXTBOOK if mode == "textbook" else abi.BP_MODE_REFERENCE
    scene = fluid_scene(bp, n, seed=8, grid_dim=grid_dim, box=(0.05 * n[0], 3.0, 0.06 * n[2]))
    outs = []
    for walk in (abi.BP_WALK_NO_STAGING, abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS):
        g = bp.ParticleSolver(scene, bp.make_params(scene, mode=m, walk_options=walk))
        g.update(1, DT, 3)
        outs.append((g.positions(), g.velocities(), g.field(abi.BP_FIELD_DENSITIES)))
        g.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("mode", ["reference", "textbook"])
@pytest.mark.parametrize("skin,iterations", [(0.0, 3), (0.0, 1), (0.004, 2)])
@pytest.mark.parametrize("name", ["one_particle", "packed", "mixed_aliased", "large", "large_aliased"])
def test_viscosity_alone_over_the_lists_is_bit_identical_to_walks(bp, gpu, name, skin, iterations, mode):
    """Pass C without the passes before it: four lanes a particle and a thread
    each, with alias classes and without, listed and queued."""
    abi = bp.abi
    m = abi.BP_MODE_TEXTBOOK if mode == "textbook" else abi.BP_MODE_REFERENCE
    if name.startswith("large"):
        scene = fluid_scene(bp, (40, 36, 34), seed=8, grid_dim=16 if name.endswith("aliased") else 64)
    else:
        scene = SCENES[name](bp)
    stages = (abi.BP_STAGE_FLUID | abi.BP_STAGE_PLANES | abi.BP_STAGE_XSPH | abi.BP_STAGE_PARTICLE_COLLISION)
    outs = []
    for walk, sk in ((abi.BP_WALK_NO_STAGING, skin), (abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS, 0.0)):
        g = bp.ParticleSolver(scene, bp.make_params(scene, mode=m, walk_options=walk, neighbor_skin=sk,
                                                    stage_mask=stages, xsph_c=0.1))
        if not walk & abi.BP_WALK_NO_LISTS and sk == 0.0:
            assert g.walk_stats(2, DT, iterations)["listed"] > 0
        else:
            g.update(2, DT, iterations)
        g.update(2, DT, iterations)
        outs.append((g.positions(), g.velocities(), g.field(abi.BP_FIELD_DENSITIES)))
        g.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("solids", [False, True])
def test_adapted_skins_of_a_bursting_block_are_bit_identical_to_walks(bp, gpu, solids):
    """A squeezed block bursting apart, where the skin grows to its widest and
    shrinks again: after every update the bits of walks without lists."""
    abi = bp.abi
    scene = (small_mixed_scene(bp, seed=7, fluid=(16, 12, 16), grid_dim=32) if solids
             else fluid_scene(bp, (16, 14, 15), seed=7, grid_dim=32, box=(3.0, 3.0, 3.0)))
    fluid = scene.phases < 0
    low = scene.positions[fluid].min(axis=0)
    scene.positions[fluid] = low + (scene.positions[fluid] - low) / np.float32(1.25)
    ways = (abi.BP_WALK_NO_STAGING, abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS)
    a, b = (bp.ParticleSolver(scene, bp.make_params(scene, mode=abi.BP_MODE_TEXTBOOK, walk_options=w)) for w in ways)
    for _ in range(12):
        for s in (a, b):
            s.update(2, DT, 3)
        np.testing.assert_array_equal(a.positions(), b.positions())
        np.testing.assert_array_equal(a.velocities(), b.velocities())
    a.close()
    b.close()


@pytest.mark.parametrize("mode", ["reference", "textbook"])
@pytest.mark.parametrize("grid_dim", [8, 32])
def test_overflowing_lists_recorded_by_each_pass(bp, gpu, grid_dim, mode):
    """The lists that every pass records for the next one (walks over the
    position records), past their capacity: the bits of walks without lists."""
    abi = bp.abi
    m = abi.BP_MODE_TEXTBOOK if mode == "textbook" else abi.BP_MODE_REFERENCE
    scene = packed(bp)
    scene.grid_dim = grid_dim
    outs = []
    for walk in (abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_PLANES, abi.BP_WALK_NO_STAGING | abi.BP_WALK_NO_LISTS):
        g = bp.ParticleSolver(scene, bp.make_params(scene, mode=m, walk_options=walk))
        for _ in range(3):
            g.update(2, DT, 4)
        outs.append((g.positions(), g.velocities(), g.field(abi.BP_FIELD_DENSITIES)))
        g.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
