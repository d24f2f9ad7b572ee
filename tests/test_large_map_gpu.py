"""The differentiable update with a depth map of more than 2^31 pixels: the voxels that project behind
that many pixels read them, and their gradients land there (a map of 64 rows with the same content is
the reference)."""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")

from luvas3d import IntegrationView, TsdfVolume  # noqa: E402
from luvas3d import grad as G  # noqa: E402
from luvas3d.camera import Intrinsics, Pose  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q8", [False, True])
def test_map_of_more_than_2_31_pixels(q8):
    W, rows = 65536, 64
    H = (1 << 31) // W + rows
    first = H - rows
    # 16 x 16 voxels of 1/8 at depth 1, one pixel apart (f = 8): every projection is an exact integer
    vol = TsdfVolume(8, 8, 0.125, (-1.0, -1.0, -0.0625), dense=(16, 16, 1), truncation=0.25, weight_q8=q8)
    rng = np.random.default_rng(4)
    part = rng.uniform(0.9, 1.1, (rows, 64)).astype(np.float32)
    packed = np.array([[oracle.pack_sample(d, (0.0, 0.0, -1.0), 0.25) for d in row] for row in part], np.uint32)
    packed[rng.random(part.shape) < 0.3] = 0  # the prior is used there
    n = vol.voxels
    wt = torch.int16 if q8 else torch.float32

    def run(height, top, width, left):
        pk = torch.zeros((height, width), dtype=torch.int32, device="cuda")
        dep = torch.zeros((height, width), device="cuda")
        pk[top:, left:left + 64] = torch.from_numpy(packed.view(np.int32)).cuda()
        dep[top:, left:left + 64] = torch.from_numpy(part).cuda()
        iv = IntegrationView(Intrinsics(8.0, 8.0, left + 20 + 7.5, top + 30 + 7.5), Pose(np.eye(3), np.array([0.0, 0.0, 1.0])),
                             5.0, None, 1.5)
        t = torch.full((n,), 0.5, device="cuda", requires_grad=True)
        w = torch.full((n,), 256 if q8 else 1, dtype=wt, device="cuda")
        prior = dep.clone() if height == rows else dep.detach()
        dep.requires_grad_(True)
        t1, w1 = G.integrate_depth(vol, iv, pk, dep, t, w, prior=prior)
        gd, gt = torch.autograd.grad(t1, (dep, t), torch.linspace(-1, 1, n, device="cuda"))
        return [a.detach().cpu().numpy() for a in (t1, w1, gd[top:, left:left + 64], gt)]

    want = run(rows, 0, 128, 30)
    assert (want[0] != 0.5).sum() > 200 and (want[2] != 0).sum() > 100
    got = run(H, first, W, W - 100)
    for a, b, name in zip(got, want, ("tsdf", "weight", "depth gradient", "tsdf gradient")):
        assert np.array_equal(a, b), name
    torch.cuda.empty_cache()
