"""Eight lanes per pixel against a thread per pixel for the storages, sums and sampled rows that
test_lanes_gpu.py leaves out: a batch that the thread kernel takes equals its views solved alone (lanes),
bit for bit."""
import numpy as np
import pytest

from helpers import arc_workload, assert_bit_equal
from luvas3d import (DTYPE_BF16, DTYPE_F16, DTYPE_F32, DTYPE_U8, FORM_EXACT, FORM_FAST, DenseStereo, SolveOptions,
                     StereoOptions)

pytestmark = pytest.mark.gpu


# 21 x 61 = 1281, 20 x 32 = 640 and 8 x 30 = 240 tiles per view (the thread kernel: above 3000, BF16, gathers
# and exact 1000)
@pytest.mark.parametrize("form,storage,compensated,variant,size,batch", [
    (FORM_FAST, DTYPE_U8, False, 14, (643, 481), 3), (FORM_FAST, DTYPE_U8, False, 30, (633, 253), 2),
    (FORM_FAST, DTYPE_BF16, False, None, (643, 481), 3), (FORM_FAST, DTYPE_BF16, True, None, (643, 481), 3),
    (FORM_FAST, DTYPE_F16, True, 14, (643, 481), 3), (FORM_FAST, DTYPE_F32, True, 30, (633, 253), 2),
    (FORM_FAST, DTYPE_F16, False, 4, (643, 481), 3), (FORM_FAST, DTYPE_F16, False, 3, (643, 481), 3),
    (FORM_FAST, DTYPE_F16, False, 2, (643, 481), 3), (FORM_EXACT, DTYPE_F32, True, 14, (633, 253), 2)])
def test_batch_equals_views_alone(form, storage, compensated, variant, size, batch):
    W, H = size
    views, imgs, _, srcs = arc_workload(n=3, W=W, H=H, f=0.875 * W)
    s = DenseStereo(W, H, views, StereoOptions(form=form, storage=storage, compensated=compensated))
    if variant is not None:
        s.variant = variant
    for i, im in enumerate(imgs):
        s.set_image(i, im)
    opts = [SolveOptions(srcs[r], 0.5, 5.0, iterations=2) for r in range(batch)]
    s.solve_all(range(batch), opts)
    want = [s.read_hypotheses_layer(r) for r in range(batch)]
    for r in range(batch):
        s.solve(r, opts[r])
        hyp, cost = s.read_hypotheses()
        assert_bit_equal(hyp, want[r][0], f"view {r} hyp")
        assert_bit_equal(cost, want[r][1], f"view {r} cost")
    assert np.isfinite(cost).all() and (cost < 0.5).mean() > 0.2
    s.destroy()


@pytest.mark.parametrize("storage", [DTYPE_F16, DTYPE_BF16])
@pytest.mark.parametrize("sources,size,batch", [(1, (250, 240), 2), (2, (633, 253), 2)])
def test_few_sources(storage, sources, size, batch):
    """One source: the thread kernel above 450 tiles, two: above 1000."""
    W, H = size
    views, imgs, _, srcs = arc_workload(n=3, W=W, H=H, f=0.875 * W)
    s = DenseStereo(W, H, views, StereoOptions(form=FORM_FAST, storage=storage))
    for i, im in enumerate(imgs):
        s.set_image(i, im)
    opts = [SolveOptions(srcs[r][:sources], 0.5, 5.0, iterations=2) for r in range(batch)]
    s.solve_all(range(batch), opts)
    want = [s.read_hypotheses_layer(r) for r in range(batch)]
    for r in range(batch):
        s.solve(r, opts[r])
        hyp, cost = s.read_hypotheses()
        assert_bit_equal(hyp, want[r][0], f"view {r} hyp")
        assert_bit_equal(cost, want[r][1], f"view {r} cost")
    s.destroy()
