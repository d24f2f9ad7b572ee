"""Surface extraction from voxel bits (csrc/mesh.cu) and its prefix sums (csrc/scan.cu) against the
oracle, bit for bit, at the sizes where they change path: grids whose rows are whole bricks (16-byte
loads) and ragged ones, f32 and Q8.8 weights, a minimum weight that is no f32, noise whose mesh falls
into many components, and scans of one tile, of several and of more tiles than the blocks add up
themselves."""
import ctypes as C

import numpy as np
import pytest

import oracle
from helpers import assert_bit_equal
from luvas3d import TsdfVolume, _lib
from luvas3d import mesh as M

pytestmark = pytest.mark.gpu


class _Array:
    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr=typestr, data=(ptr, False), version=3,
                                             strides=None)


def _fill(volume, tsdf, weight):
    import torch

    t, w = C.c_void_p(), C.c_void_p()
    _lib.check(_lib.load().l3d_tsdf_device_buffers(volume._h(), C.byref(t), C.byref(w)))
    volume.synchronize()
    torch.as_tensor(_Array(t.value, tsdf.size, "<f4"), device="cuda").copy_(torch.from_numpy(tsdf.reshape(-1)))
    kind = "<i2" if weight.dtype == np.uint16 else "<f4"
    flat = weight.reshape(-1)
    torch.as_tensor(_Array(w.value, weight.size, kind), device="cuda").copy_(
        torch.from_numpy(flat.view(np.int16) if weight.dtype == np.uint16 else flat))
    torch.cuda.synchronize()


@pytest.mark.parametrize("dims", [(8, 8, 8), (16, 8, 24), (13, 9, 17), (20, 30, 11), (40, 1, 40)])
@pytest.mark.parametrize("q8", [False, True])
def test_dense_surface_equals_oracle(dims, q8):
    X, Y, Z = dims
    rng = np.random.default_rng(X * 10000 + Y * 100 + Z)
    tsdf = rng.normal(size=(Z, Y, X)).astype(np.float32)
    tsdf[rng.random(tsdf.shape) < 0.05] = -0.0  # not negative
    steps = rng.integers(1, 6, size=tsdf.shape)  # weights 0.1 .. 0.5, or the Q8.8 values around them
    weight = np.round(steps * 25.6).astype(np.uint16) if q8 else (steps * 0.1).astype(np.float32)
    weight[rng.random(tsdf.shape) < 0.03] = 0
    origin, voxel = (-0.3, 0.1, 2.0), 0.013
    vol = TsdfVolume(8, 8, voxel, origin, dense=dims, weight_q8=q8)
    _fill(vol, tsdf, weight)
    nb = [(d + 7) // 8 for d in dims]
    pad = [(0, n * 8 - d) for n, d in zip(nb[::-1], dims[::-1])]
    # the oracle's pool: voxels outside the grid unobserved
    def bricks(a, fill):
        p = np.pad(a, pad, constant_values=fill).reshape(nb[2], 8, nb[1], 8, nb[0], 8)
        return np.ascontiguousarray(p.transpose(0, 2, 4, 1, 3, 5)).reshape(-1)
    wf = weight.astype(np.float32) * (1 / 256 if q8 else 1)
    lookup = np.arange(nb[0] * nb[1] * nb[2], dtype=np.int32)
    for minimum in (0.0, 0.1, 0.2):  # 0.1 and 0.2 are no f32 and lie beside the weights
        got = M.extract_surface(vol, minimum)
        pos, nrm, idx = oracle.extract_surface(origin, voxel, nb, lookup, bricks(tsdf, 1.0),
                                               bricks(wf, -1.0), minimum)
        assert_bit_equal(got.positions, pos, "positions")
        assert_bit_equal(got.normals, nrm, "normals")
        np.testing.assert_array_equal(got.indices, idx)


def test_noise_components_equal_oracle():
    rng = np.random.default_rng(5)
    dims = (48, 40, 56)
    tsdf = np.where(rng.random((56, 40, 48)) < 0.06, -1.0, 1.0).astype(np.float32)
    vol = TsdfVolume(8, 8, 0.01, (0, 0, 0), dense=dims)
    _fill(vol, tsdf, np.ones_like(tsdf))
    m = M.extract_surface_device(vol, 0.5)
    base = m.read()
    assert base.indices.size > 30000
    for fraction, least in ((0.0, 1), (0.0, 9), (0.0, 13), (0.0, 40), (2.0, 1)):
        r = m.remove_small_components(fraction, least)
        got = r.read()
        p, n, i = oracle.remove_small_components(base.positions, base.normals, base.indices, fraction, least)
        assert_bit_equal(got.positions, p, "positions")
        assert_bit_equal(got.normals, n, "normals")
        np.testing.assert_array_equal(got.indices, i)


@pytest.mark.parametrize("cells", [(1, 1, 1), (2047, 1, 1), (16, 16, 8), (2049, 1, 1), (131, 127, 127)])
def test_brick_grid_scan_sizes_equal_oracle(cells):
    rng = np.random.default_rng(sum(cells))
    voxel = 0.01
    extent = [c * 8 * voxel - voxel for c in cells]
    pts = (rng.random((4000, 3)) * extent).astype(np.float32)
    got = M.brick_grid((0, 0, 0), voxel, extent, pts, 0.004)
    want = oracle.brick_grid((0, 0, 0), voxel, extent, pts, 0.004)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
