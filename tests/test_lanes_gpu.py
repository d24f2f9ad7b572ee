"""The propagate step with eight lanes per pixel against the one with a thread per pixel: a batch large
enough for the thread kernel equals its views solved alone (lanes), bit for bit, at sizes that leave
partial tiles on both edges.  Both walk patchmatch.wgsl.ts:349-423 in the same order of candidates, so
planes, costs and packed maps are equal; a wrong tie between equal candidates, a lane's refinement in
another place or a write from a lane outside the image would show."""
import numpy as np
import pytest

from helpers import arc_workload, assert_bit_equal
from luvas3d import DTYPE_F16, DTYPE_F32, FORM_EXACT, FORM_FAST, DenseStereo, SolveOptions, StereoOptions

pytestmark = pytest.mark.gpu


# 128-pixel tiles of one colour per view: 21 x 61 = 1281 and 20 x 32 = 640; the thread kernel starts
# above 3000 (filtered samples) and 1000 (gathers, exact) tiles
@pytest.mark.parametrize("form,storage,variant,size,batch", [
    (FORM_FAST, DTYPE_F16, 14, (643, 481), 3), (FORM_FAST, DTYPE_F32, 30, (633, 253), 2),
    (FORM_EXACT, DTYPE_F32, 14, (633, 253), 2)])
@pytest.mark.parametrize("geometric", [False, True])
def test_batch_equals_views_alone(form, storage, variant, size, batch, geometric):
    W, H = size
    views, imgs, truth, srcs = arc_workload(n=3, W=W, H=H, f=0.875 * W)
    s = DenseStereo(W, H, views, StereoOptions(form=form, storage=storage))
    s.variant = variant
    for i, im in enumerate(imgs):
        s.set_image(i, im)
    opts = [SolveOptions(srcs[r], 0.5, 5.0, iterations=2) for r in range(batch)]
    geo = [SolveOptions(srcs[r], 0.5, 5.0, iterations=1, geometric=True) for r in range(batch)]
    s.solve_all(range(batch), opts)
    if geometric:
        before = [s.depth_map(r) for r in range(3)]
        s.solve_all(range(batch), geo)
    want = [(*s.read_hypotheses_layer(r), s.depth_map(r)) for r in range(batch)]
    for r in range(batch):
        if geometric:  # a batch reads the maps as they were when it started
            for k in range(3):
                s.write_depth_map(k, before[k])
        s.solve(r, geo[r] if geometric else opts[r])
        hyp, cost = s.read_hypotheses()
        assert_bit_equal(hyp, want[r][0], f"view {r} hyp")
        assert_bit_equal(cost, want[r][1], f"view {r} cost")
        assert np.array_equal(s.depth_map(r), want[r][2]), f"view {r} packed"
