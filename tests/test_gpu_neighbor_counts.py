"""Neighbour counts on caller buffers against the oracle, where columns wrap
around the table and around the occupancy at which longer trips are taken."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_grid import gpu_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [0.2, 0.07])
@pytest.mark.parametrize("n,D,spread", [
    (1, 4, 1.0), (33, 4, 1.0), (383, 4, 0.5), (384, 4, 0.5), (5000, 4, 2.0),  # most columns wrap
    (3071, 8, 1.0), (3072, 8, 1.0), (3073, 8, 3.0),
    (60_000, 32, 2.5),   # below 65,536 particles, columns of both kinds in a warp
    (90_000, 32, 5.0), (100_003, 16, 1.6),
])
def test_counts_of_wrapping_columns_match_the_oracle(bp, gpu, oracle, n, D, spread, h):
    pos = np.random.default_rng(n + D).uniform(-spread, spread, (n, 3)).astype(np.float32)
    _, _, order, start, end, counts, _ = gpu_grid(bp, gpu, pos, 0.2, D, h)
    np.testing.assert_array_equal(counts, oracle.neighbor_counts("oracle", pos[order], 0.2, D, h, start, end))
