"""A recording that takes over the buffers and graphs of an ended one gives the
gradients of a fresh solver's."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import fluid_scene

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def record(s, params, frames, iterations, every, weights):
    s.set_params(params)
    s.tape_begin(every)
    for _ in range(frames):
        s.update(2, DT, iterations)
    out = s.backward(weights, 0.1 * weights)
    s.tape_end()
    return out


@pytest.mark.parametrize("kind", ["flag", "fluid"])
def test_recordings_after_one_another_match_fresh_solvers(bp, gpu, kind):
    """Other lengths, checkpoint spacings, iteration counts and parameters from
    one recording to the next, a recording begun over an open one and plain
    updates between: each from the same snapshot as a fresh solver's."""
    abi = bp.abi
    if kind == "flag":
        scene = bp.scenes.flag_scene(n=12)
        base = dict(mode=abi.BP_MODE_TEXTBOOK, wind_drag=1.0, wind_lift=0.3, mass_scaling_k=0.0,
                    stage_mask=abi.BP_STAGE_PLANES | abi.BP_STAGE_WIND | abi.BP_STAGE_DISTANCE
                    | abi.BP_STAGE_IMMOVABLE)
        steps = [(dict(wind_velocity=(4.0, 0.0, 0.0)), 3, 4, 2), (dict(wind_velocity=(1.0, 0.0, 2.0)), 5, 2, 10),
                 (dict(wind_velocity=(4.0, 0.0, 0.0)), 2, 4, 1)]
    else:
        scene = fluid_scene(bp, (6, 6, 6), seed=2, grid_dim=16)
        base = dict(stage_mask=abi.BP_STAGE_FLUID | abi.BP_STAGE_PLANES | abi.BP_STAGE_XSPH)
        steps = [(dict(), 2, 3, 2), (dict(xsph_c=0.01), 3, 3, 10), (dict(), 2, 2, 1)]
    weights = np.random.default_rng(1).normal(size=(scene.num_particles, 3)).astype(np.float32)
    s = bp.ParticleSolver(scene, bp.make_params(scene, **base))
    begin = s.snapshot()
    for k, (over, frames, iterations, every) in enumerate(steps):
        params = bp.make_params(scene, **{**base, **over})
        if k == 1:
            s.tape_begin(1)
            s.update(2, DT, iterations)
            s.tape_begin(1)  # over an open recording
            s.update(2, DT, 1)
            s.tape_end()
        s.update(2, DT, 3)
        s.restore(begin)
        got = record(s, params, frames, iterations, every, weights)
        fresh = bp.ParticleSolver(scene, params)
        want = record(fresh, params, frames, iterations, every, weights)
        np.testing.assert_array_equal(s.positions(), fresh.positions())
        fresh.close()
        for name in want:
            np.testing.assert_array_equal(got[name], want[name], err_msg=name)
    s.close()
