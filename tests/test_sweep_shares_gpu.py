"""The sweep's hand-out of passes to warps (k_integrate_many_list), where its rule changes: as many passes as
warps or fewer, a few rounds by the warps' numbers, then asking for one pass a share, two or three (of 4
and 2 and 13 of 16 a brick), a whole brick; at once and in the slabs of a read-back.  Every brick is kept,
and the volume equals the views integrated one by one."""
import numpy as np
import pytest

import oracle
from helpers import assert_bit_equal
from luvas3d import IntegrationView, TsdfVolume
from luvas3d.camera import Intrinsics, look_at

pytestmark = pytest.mark.gpu


# 4736 warps (148 SMs); 4 passes a brick where the rows are multiples of four, else 16
@pytest.mark.parametrize("dims", [(64, 64, 64), (72, 64, 64), (104, 104, 104), (128, 128, 128), (216, 216, 216), (248, 248, 248),
                                  (288, 288, 280), (61, 37, 55), (66, 66, 66), (101, 99, 101), (135, 133, 131), (253, 251, 249)])
@pytest.mark.parametrize("q8", [False, True])
def test_sweep_equals_views_one_by_one(dims, q8):
    voxel = 2.0 / max(dims)
    k = Intrinsics(110.0, 110.0, 64.0, 48.0)
    views = [IntegrationView(k, look_at(eye, (0, 0, 0)), 20.0, None, c)
             for eye, c in (((0.3, 0.2, -4.2), 0.0), ((3.9, -0.4, 1.0), 1.5))]
    rng = np.random.default_rng(dims[0])
    depths = rng.uniform(3.0, 7.0, (2, 96, 128))
    maps = np.array([[[oracle.pack_sample(d, (0.0, 0.0, -1.0), 0.3) for d in row] for row in m] for m in depths], np.uint32)
    origin = tuple(-voxel * d / 2 for d in dims)
    a, b, c = (TsdfVolume(128, 96, voxel, origin, dense=dims, truncation=2.0, weight_q8=q8) for _ in range(3))
    for v, m in zip(views, maps):
        a.integrate(v, depth=m)
    b.integrate_many(views, depths=maps)
    want, weight = a.read()
    assert (weight > 0).mean() > 0.7
    for t, w in (b.read(), c.integrate_many_read(views, depths=maps)):
        assert_bit_equal(t.reshape(-1), want.reshape(-1), "tsdf")
        assert_bit_equal(w.reshape(-1), weight.reshape(-1), "weight")
    for v in (a, b, c):
        v.destroy()
