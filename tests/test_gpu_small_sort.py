"""The one-launch hash and sort of small inputs (one cluster of CTAs) against
a stable sort of the oracle's cell ids, at the edges of its tiles and items."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid_dim", [4, 64, 512])
@pytest.mark.parametrize("n", [1, 511, 512, 513, 4096, 4097, 8193, 16385, 32768, 32769, 65535, 65536, 65537])
def test_small_grid_build_matches_a_stable_sort(bp, gpu, oracle, n, grid_dim):
    torch, lib = gpu, bp.abi.load()
    rng = np.random.default_rng(n + grid_dim)
    pos = rng.uniform(-3.0, 3.0, (n, 3)).astype(np.float32)  # crowded cells on every table: ties
    cell = 0.2
    ids, want_sorted, want_order, start, end = oracle.grid_build("oracle", pos, cell, grid_dim)
    p = torch.from_numpy(pos).cuda()
    i32 = dict(dtype=torch.int32, device="cuda")
    out = [torch.empty(n, **i32) for _ in range(3)] + [torch.full((grid_dim ** 3,), -1, **i32) for _ in range(2)]
    size = C.c_size_t()
    bp.abi.check(lib, lib.bp_grid_workspace_size(n, grid_dim, C.byref(size)))
    ws = torch.empty(size.value, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    bp.abi.check(lib, lib.bp_grid_build(stream, n, p.data_ptr(), C.c_float(cell), grid_dim,
                                        *[t.data_ptr() for t in out], ws.data_ptr(), size.value))
    for got, want in zip(out, (ids, want_sorted, want_order, start, end)):
        np.testing.assert_array_equal(got.cpu().numpy(), want)
