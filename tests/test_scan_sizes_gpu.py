"""Prefix sums of thousands of tiles (csrc/scan.cu), whose own sums take a block several steps: brick grids of
whole and partial steps against the oracle."""
import numpy as np
import pytest

import oracle
from luvas3d import mesh as M

pytestmark = pytest.mark.gpu


# tiles of 2048 cells; 2048 tiles a step: one step, one and two cells, five less a bit
@pytest.mark.parametrize("cells", [(256, 128, 128), (699051, 6, 1), (151, 149, 932)])
def test_brick_grids_of_many_tiles_equal_oracle(cells):
    rng = np.random.default_rng(sum(cells))
    voxel = 0.01
    extent = [c * 8 * voxel - voxel for c in cells]
    pts = (rng.random((20000, 3)) * extent).astype(np.float32)
    got = M.brick_grid((0, 0, 0), voxel, extent, pts, 0.004)
    assert tuple(got[0]) == cells
    want = oracle.brick_grid((0, 0, 0), voxel, extent, pts, 0.004)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
