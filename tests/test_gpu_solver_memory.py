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


@pytest.mark.parametrize("kind", ["single", "batch"])
def test_shorter_lists_where_memory_is_short(bp, gpu, tmp_path, kind):
    """Where the lists of 384 entries do not fit, and those of 192 do not
    either, the solver is created with the next capacity: the same results, in
    fluid whose lists overflow under all three; where none fits, the error."""
    run_child(tmp_path, f"""
        scene = fluid_scene(bp, (14, 12, 10), seed=4, grid_dim=16)
        x = scene.positions
        c = x.mean(axis=0)
        core = np.all(np.abs(x - c) < 0.35, axis=1)
        x[core] = c + (x[core] - c) * np.float32(0.4)
        n = scene.num_particles
        if {kind!r} == "single":
            make = lambda: bp.ParticleSolver(scene, bp.make_params(scene))
        else:
            make = lambda: bp.BatchSolver([scene, scene], [bp.make_params(scene)] * 2)
            n *= 2
        outs = []
        for above in (0, 4 * 384 * n - 1, 4 * 192 * n - 1):
            arm(0, above)
            g = make()
            arm()
            for _ in range(3):
                g.step(1.0 / 60.0, 2, 3)
            outs.append((g.positions(), g.velocities()))
            g.close()
        for out in outs[1:]:
            for a, b in zip(outs[0], out):
                np.testing.assert_array_equal(a, b)
        arm(0, 4 * 144 * n - 1)
        try:
            make()
            raise SystemExit("created")
        except Exception as e:
            assert "status 3" in str(e), e  # BP_ERR_OUT_OF_MEMORY
        arm()
        make().close()
        """)
