"""A solver's hash and sort, in one launch and in a chain of them, against the
oracle's grid of the predicted positions."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid_dim", [8, 64, 128])  # one, two and three passes
@pytest.mark.parametrize("n", [32767, 32768, 32769, 65536, 65537])
def test_sorted_order_matches_the_oracle(bp, gpu, oracle, n, grid_dim):
    """Around the sizes where the launches change: cell ids in sorted order and
    the original index of each sorted particle after a substep that only moves
    particles to where they were predicted."""
    abi = bp.abi
    rng = np.random.default_rng(n + grid_dim)
    s = bp.scenes.Scene(name="drift")
    s.particle_radius, s.kernel_radius, s.cell_size, s.grid_dim = 0.05, 0.2, 0.2, grid_dim
    s._append(rng.uniform(-3.0, 3.0, (n, 3)), 1.0, np.full(n, -1))
    s.velocities = rng.uniform(-1.0, 1.0, (n, 3)).astype(np.float32)
    g = bp.ParticleSolver(s, bp.make_params(s, stage_mask=0))
    g.update(1, 1.0 / 120.0, 0)
    _, cells, order, _, _ = oracle.grid_build("oracle", g.positions(), 0.2, grid_dim)
    np.testing.assert_array_equal(g.field(abi.BP_FIELD_SORTED_CELL_IDS), cells)
    np.testing.assert_array_equal(g.field(abi.BP_FIELD_MAP_TO_ORIGINAL), order)
    g.close()
