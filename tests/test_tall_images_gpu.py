"""The plain form on images taller than a launch's blocks along one axis cover (131070 rows): planes and
costs equal the oracle bit for bit.  (An upload converts at most 65535 rows, so the images are written into
the handle's device buffer.)"""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")

from helpers import assert_bit_equal  # noqa: E402
from luvas3d import DenseStereo, SolveOptions  # noqa: E402
from luvas3d.camera import Intrinsics, Pose, StereoView  # noqa: E402

pytestmark = pytest.mark.gpu


class _Array:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f4", data=(ptr, False), version=3, strides=None)


@pytest.mark.parametrize("H", [131070, 131071, 131080])
def test_tall_plain_solve_equals_oracle(H):
    W = 16
    k = Intrinsics(900.0, 900.0, W / 2, H / 2)
    views = [StereoView(k, Pose(np.eye(3), np.array([0.0, y, 0.0]))) for y in (0.0, 0.05, -0.04)]
    rng = np.random.default_rng(H)
    rows = np.repeat(rng.integers(0, 256, (3, (H + 3) // 4, W)), 4, axis=1)[:, :H]
    images = (rows / 255.0).astype(np.float32)
    s = DenseStereo(W, H, views)
    o = oracle.Stereo(W, H, views, images, 32)
    torch.as_tensor(_Array(s.buffers().images, images.size), device="cuda").copy_(torch.from_numpy(images.reshape(-1)))
    torch.cuda.synchronize()
    s.solve(0, SolveOptions([1, 2], 0.5, 3.0, iterations=1))
    o.solve(0, [1, 2], min_depth=0.5, max_depth=3.0, iterations=1)
    hyp, cost = s.read_hypotheses()
    assert (cost[-12:] < 2.0).any()  # matches in the last rows
    assert_bit_equal(cost.reshape(-1), o.cost.reshape(-1), "cost")
    assert_bit_equal(hyp.reshape(-1), o.hyp.reshape(-1), "planes")
    s.destroy()
