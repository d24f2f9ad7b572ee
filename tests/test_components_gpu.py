"""removeSmallComponents (mesh.ts:37-87) of meshes whose labels form long chains: one component of several
hundred thousand faces among small ones, removed many times over, equals the oracle every time."""
import numpy as np
import pytest

import oracle
from helpers import assert_bit_equal
from luvas3d import mesh as M

pytestmark = pytest.mark.gpu


def _pool(tsdf):
    """A host volume of all the bricks of a dense array (z, y, x), every voxel observed."""
    nz, ny, nx = (d // 8 for d in tsdf.shape)
    bricks = tsdf.reshape(nz, 8, ny, 8, nx, 8).transpose(0, 2, 4, 1, 3, 5)
    return dict(origin=(0.0, 0.0, 0.0), voxel=0.01, dims=(nx, ny, nz),
                lookup=np.arange(nx * ny * nz, dtype=np.int32),
                tsdf=np.ascontiguousarray(bricks, np.float32).reshape(-1),
                weight=np.ones(tsdf.size, np.float32))


@pytest.mark.parametrize("shape", ["gyroid", "sheets"])
def test_large_components_survive_every_time(shape):
    z, y, x = np.meshgrid(*[np.arange(128, dtype=np.float32)] * 3, indexing="ij", sparse=True)
    if shape == "gyroid":  # one component
        a = 0.33
        tsdf = np.sin(a * x) * np.cos(a * y) + np.sin(a * y) * np.cos(a * z) + np.sin(a * z) * np.cos(a * x)
    else:  # flat ones, seven voxels apart
        tsdf = np.abs(x % 14 - 6.7) - 3.3 + 0 * (y + z)
    tsdf = tsdf.astype(np.float32)
    rng = np.random.default_rng(1)
    tsdf[rng.random(tsdf.shape) < 2e-4] *= -1  # specks
    m = M.extract_surface_device(_pool(np.clip(tsdf, -1, 1)), 0.5)
    base = m.read()
    faces = base.indices.size // 3
    p, n, i = oracle.remove_small_components(base.positions, base.normals, base.indices, 0.0, 1000)
    assert 100000 < i.size // 3 < faces
    for _ in range(100):
        r = m.remove_small_components(0.0, 1000)
        got = r.read()
        r.destroy()
        np.testing.assert_array_equal(got.indices, i)
        assert_bit_equal(got.positions, p, "positions")
        assert_bit_equal(got.normals, n, "normals")
    m.destroy()
