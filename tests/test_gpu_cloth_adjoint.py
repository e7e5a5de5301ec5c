"""The adjoint of a cloth iteration's end in one launch against the launches it
replaces."""
from __future__ import annotations

import copy

import numpy as np
import pytest

from test_gpu_cloth_step import cloth

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


@pytest.mark.parametrize("iterations", [1, 4])
@pytest.mark.parametrize("n,pinned", [(2, True), (3, False), (11, True), (33, True)])
def test_cloth_step_gradients_match_the_separate_launches(bp, gpu, n, pinned, iterations):
    """The same cloth (a doubled edge, one of no length, one from a particle to
    itself) alone and among four times as many loose particles far away, which
    no stage couples to it: there the edges, their sums, the pins and the planes
    are launches of their own.  Both add the same terms in the same order, so
    what differs is how the compiler contracts them: 16 operations an edge, 14
    edges and 16 iterations of 6e-8 each come to 4e-6 as random steps."""
    abi = bp.abi
    alone = cloth(bp, n, pinned)
    m = alone.num_particles
    among = copy.deepcopy(alone)
    rng = np.random.default_rng(2)
    among._append(rng.uniform(20.0, 24.0, (4 * m, 3)), 1.0, among._solid_phases(4 * m, False))
    among.velocities[m:] = 0.0
    stages = (abi.BP_STAGE_PLANES | abi.BP_STAGE_WIND | abi.BP_STAGE_DISTANCE | abi.BP_STAGE_IMMOVABLE)
    weights = rng.normal(size=(5 * m, 3)).astype(np.float32)
    outs = []
    for scene in (alone, among):
        k = scene.num_particles
        g = bp.ParticleSolver(scene, bp.make_params(scene, mode=abi.BP_MODE_TEXTBOOK, stage_mask=stages,
                                                    wind_velocity=(4.0, 0.0, 1.0), wind_drag=1.0, wind_lift=0.3,
                                                    mass_scaling_k=0.0))
        w = np.zeros((k, 3), np.float32)
        w[:m] = weights[:m]
        g.tape_begin(3)
        for _ in range(2):
            g.update(2, DT, iterations)
        outs.append(dict(g.backward(w, 0.1 * w), x=g.positions()))
        g.close()
    for name, a in outs[0].items():
        b = outs[1][name][:m] if name in ("positions", "velocities", "x") else outs[1][name]
        assert np.isfinite(a).all()
        np.testing.assert_allclose(a, b, rtol=0.0, atol=2e-5 * max(float(np.abs(a).max()), 1e-30), err_msg=name)
