"""Device memory a solver asks for."""
from __future__ import annotations

import pytest

from test_gpu_recording_memory import run_child

pytestmark = pytest.mark.gpu


def test_verlet_lists_take_memory_only_where_walks_read_them(bp, gpu, tmp_path):
    """1 KB a particle where a skin is asked of walks that keep Verlet lists:
    not of those that take the skin for the substep lists, until other walks
    are set, and then with the results of the others."""
    run_child(tmp_path, """
        scene = fluid_scene(bp, (16, 12, 10), seed=4, grid_dim=16)
        lists = 1024 * scene.num_particles

        def taken(f):
            arm()
            return f(), shim.shim_bytes()

        walks = [bp.make_params(scene, walk_options=w, neighbor_skin=k)
                 for w, k in ((abi.BP_WALK_NO_STAGING, 0.0), (abi.BP_WALK_NO_STAGING, 0.1), (0, 0.1))]
        (plain, least), (skin, same), (staged, most) = [taken(lambda: bp.ParticleSolver(scene, p)) for p in walks]
        assert same == least, (least, same)
        assert most >= least + lists, (least, most)
        assert taken(lambda: skin.set_params(walks[2]))[1] == most - least
        for g in (plain, skin, staged):
            g.update(2, 1.0 / 60.0, 3)
        for g in (skin, staged):
            np.testing.assert_array_equal(g.positions(), plain.positions())
        """)
