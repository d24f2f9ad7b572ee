"""Targets of l3d_mesh_read and l3d_cloud_read: pageable, pinned and managed host memory receive the same
bytes, and a device pointer is left to the CUDA runtime's copy, which takes it or refuses it with a
status; the process and later reads are unharmed either way."""
import ctypes as C

import numpy as np
import pytest

from luvas3d import _lib
from luvas3d import mesh as M
from luvas3d.cloud import PointAccumulator
from mesh_fixtures import sphere_volume

pytestmark = pytest.mark.gpu


def _cloud():
    rng = np.random.default_rng(3)
    s = np.zeros((40000, 9))  # 41 bytes a point: more than one buffer of 1 MB
    ids = rng.choice(100 ** 3, len(s), replace=False)
    s[:, :3] = (np.stack([ids % 100, ids // 100 % 100, ids // 10000], 1) + 0.5) * 0.01
    s[:, 5] = 1.0
    acc = PointAccumulator(0.01)
    acc.add_points(s)
    c = acc.cloud()

    def read(p):
        n = C.c_int64()
        return _lib.load().l3d_cloud_read(acc._h(), 1, len(s), C.byref(n), p, None, None, None, None)
    return read, c.positions, acc


def _mesh():
    m = M.extract_surface_device(sphere_volume(), 0.5)
    return lambda p: _lib.load().l3d_mesh_read(m._handle, p, None, None), m.read().positions, m


@pytest.mark.parametrize("source", [_cloud, _mesh])
@pytest.mark.parametrize("kind", ["pinned", "managed", "device"])
def test_reads_into_memory_that_cuda_knows(source, kind):
    import torch

    read, want, keep = source()
    flat = want.reshape(-1)
    if kind == "managed":
        rt = C.CDLL("libcudart.so.12")
        p = C.c_void_p()
        assert rt.cudaMallocManaged(C.byref(p), C.c_size_t(flat.nbytes), C.c_uint(1)) == 0
        assert read(p) == 0
        got = np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_float)), (flat.size,)).copy()
        assert rt.cudaFree(p) == 0
    else:
        t = torch.zeros(flat.size, dtype=torch.float32, **({"pin_memory": True} if kind == "pinned" else {"device": "cuda"}))
        torch.cuda.synchronize()
        rc = read(C.c_void_p(t.data_ptr()))
        assert rc == 0 or kind == "device"
        got = t.cpu().numpy() if rc == 0 else flat
    assert np.array_equal(got.view(np.uint32), flat.view(np.uint32))
    again = np.zeros_like(flat)
    assert read(_lib.ptr(again)) == 0
    assert np.array_equal(again.view(np.uint32), flat.view(np.uint32))
    keep.destroy()

