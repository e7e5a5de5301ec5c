"""That the scenes on which substep lists are compared with walks take them."""
from __future__ import annotations

import pytest

from conftest import fluid_scene, small_mixed_scene
from test_gpu_lists import grains
from test_gpu_solver import contact_scene

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def outside(bp, n):
    return fluid_scene(bp, n, seed=8, grid_dim=64, box=(0.05 * n[0], 3.0, 0.06 * n[2]))


SCENES = {
    **{f"side_{k}": (lambda bp, k=k: fluid_scene(bp, (k,) * 3, seed=k, grid_dim=64, box=(4.0, 4.0, 4.0)))
       for k in (24, 31, 36)},
    "bursting": lambda bp: fluid_scene(bp, (16, 14, 15), seed=7, grid_dim=32, box=(3.0, 3.0, 3.0)),
    "bursting_solids": lambda bp: small_mixed_scene(bp, seed=7, fluid=(16, 12, 16), grid_dim=32),
}


@pytest.mark.parametrize("mode", ["reference", "textbook"])
@pytest.mark.parametrize("name", list(SCENES))
def test_most_reads_are_from_lists(bp, gpu, name, mode):
    """Of two substeps with three iterations and the post passes: three reads a
    fluid particle and substep, most of them served by its list."""
    abi = bp.abi
    m = abi.BP_MODE_TEXTBOOK if mode == "textbook" else abi.BP_MODE_REFERENCE
    scene = SCENES[name](bp)
    g = bp.ParticleSolver(scene, bp.make_params(scene, mode=m))
    stats = g.walk_stats(2, DT, 3)
    g.close()
    assert stats["listed"] > 3 * int((scene.phases < 0).sum()), stats


@pytest.mark.parametrize("mode", ["reference", "textbook"])
@pytest.mark.parametrize("n", [(20, 12, 16), (40, 36, 20), (40, 36, 34)])
def test_blocks_outside_their_box_read_lists_and_walk(bp, gpu, n, mode):
    abi = bp.abi
    m = abi.BP_MODE_TEXTBOOK if mode == "textbook" else abi.BP_MODE_REFERENCE
    scene = outside(bp, n)
    g = bp.ParticleSolver(scene, bp.make_params(scene, mode=m))
    stats = g.walk_stats(1, DT, 3)
    g.close()
    assert stats["listed"] > 0 and stats["cells_no_list"] > scene.num_particles, stats


def test_a_batch_with_solids_reads_lists(bp, gpu):
    scenes = [contact_scene(bp, seed=2), fluid_scene(bp, (8, 8, 8), seed=6, grid_dim=32), grains(bp)]
    g = bp.BatchSolver(scenes, [bp.make_params(s, rest_density=1000.0) for s in scenes])
    stats = g.walk_stats(2, DT, 3)
    g.close()
    assert stats["listed"] > g.n, stats
