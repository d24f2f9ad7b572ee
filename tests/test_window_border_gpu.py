"""Windows whose warped samples land on, just inside or just outside a source's border, bit for bit
against the FP32 oracle: hypothesis_cost (patchmatch.wgsl.ts:192-233) of planes under cameras that
differ by whole pixels, by a rounding of one, and by a half turn.  The kernels decide from the four
corners whether a window's samples need their own tests; a bound that is too tight or a rejected
corner that the per-sample arithmetic accepts would change these costs."""
import numpy as np
import pytest

import oracle
from helpers import assert_bit_equal
from luvas3d import FORM_EXACT, FORM_PLAIN, DenseStereo, SolveOptions, StereoOptions
from luvas3d.camera import Intrinsics, Pose, StereoView

pytestmark = pytest.mark.gpu


def _views(W, H, f):
    k = Intrinsics(f, f, W / 2, H / 2)
    turn = np.diag([-1.0, 1.0, -1.0])
    shift = [(0, 0, 0), (8 / f, 0, 0), (-4 / f, 2 / f, 0), (1e-7, -1e-7, 0), (0, 0, 0.25)]
    views = [StereoView(k, Pose(np.eye(3), np.array(t, dtype=np.float64))) for t in shift]
    return views + [StereoView(k, Pose(turn, np.zeros(3)))]


@pytest.mark.parametrize("size", [(11, 11), (12, 13), (33, 16), (64, 48), (2049, 13)])
@pytest.mark.parametrize("form", [FORM_EXACT, FORM_PLAIN])
def test_plane_cost_at_borders_bit_exact(size, form):
    W, H = size
    f = 64.0
    views = _views(W, H, f)
    rng = np.random.default_rng(W * 1000 + H)
    imgs = [rng.random((H, W)).astype(np.float32) for _ in views]
    srcs = list(range(1, len(views)))
    o = oracle.Stereo(W, H, views, imgs, 32)
    s = DenseStereo(W, H, views, StereoOptions(form=form))
    for i, im in enumerate(imgs):
        s.set_image(i, im)
    kw = dict(min_depth=0.05, max_depth=1e30)
    # fronto-parallel planes at depths that move samples by whole pixels, tilted planes around
    # them, and planes so far or so tilted that positions leave the ordinary range
    for kind in range(4):
        planes = np.zeros((H, W, 4), dtype=np.float32)
        tilt = (0.0, 1e-6, 0.5, 3.0)[kind]
        n = rng.normal(size=(H, W, 3)) * tilt + np.array([0, 0, -1.0])
        planes[..., :3] = n / np.linalg.norm(n, axis=-1, keepdims=True)
        planes[..., 3] = rng.choice([0.125, 0.25, 0.5, 1.0, 2.0, 4.0, 1e6, 1e25], size=(H, W))
        want, _ = o.plane_cost(0, srcs, planes, **kw)
        got = s.plane_cost(0, SolveOptions(srcs, **kw), planes)
        assert_bit_equal(got, want.astype(np.float32), f"hypothesis cost, tilt {tilt}")


@pytest.mark.parametrize("size", [(13, 11), (46, 31)])
@pytest.mark.parametrize("form", [FORM_EXACT, FORM_PLAIN])
def test_solve_near_borders_bit_exact(size, form):
    """Whole solves on images so small that every window is near a border."""
    W, H = size
    views = _views(W, H, 64.0)
    rng = np.random.default_rng(W)
    base = rng.random((H + 16, W + 16)).astype(np.float32)
    imgs = [np.ascontiguousarray(base[8 - i:8 - i + H, 8 + i:8 + i + W]) for i in range(len(views))]
    srcs = list(range(1, len(views)))
    o = oracle.Stereo(W, H, views, imgs, 32)
    s = DenseStereo(W, H, views, StereoOptions(form=form))
    for i, im in enumerate(imgs):
        s.set_image(i, im)
    o.solve(0, srcs, min_depth=0.1, max_depth=8.0, iterations=2)
    s.solve(0, SolveOptions(srcs, 0.1, 8.0, iterations=2))
    hyp, cost = s.read_hypotheses()
    assert_bit_equal(hyp, o.hyp, "hyp")
    assert_bit_equal(cost, o.cost, "cost")


@pytest.mark.parametrize("size", [(12, 13), (33, 16), (64, 48)])
def test_gradient_cost_at_borders_matches_plane_cost(size):
    """The gradient kernel's forward cost of fronto-parallel planes (angles 0) is the sum of the plain
    form's view costs: the same positions, so the same windows are lost (their cost, 2, is far from any
    other by more than the tolerance), and the same FP32 sums but for the homography's composition
    (1e-4 per source is the forward cost's tolerance elsewhere)."""
    import torch

    from luvas3d import grad

    W, H = size
    views = _views(W, H, 64.0)
    rng = np.random.default_rng(W)
    imgs = [rng.random((H, W)).astype(np.float32) for _ in views]
    srcs = list(range(1, len(views)))
    s = DenseStereo(W, H, views)
    for i, im in enumerate(imgs):
        s.set_image(i, im)
    planes = np.zeros((H, W, 4), dtype=np.float32)
    planes[..., 2] = -1.0
    planes[..., 3] = rng.choice([0.125, 0.25, 0.5, 1.0, 2.0, 4.0], size=(H, W))
    _, vc = s.plane_cost(0, SolveOptions(srcs, 0.05, 1e30), planes, view_costs=True)
    pl = torch.zeros((H, W, 3), device="cuda")
    pl[..., 0] = torch.from_numpy(planes[..., 3]).cuda()
    got = grad.ncc_cost(s, 0, srcs, pl.contiguous()).cpu().numpy()
    np.testing.assert_allclose(got, vc[..., :len(srcs)].sum(-1), rtol=0, atol=1e-4 * len(srcs))
