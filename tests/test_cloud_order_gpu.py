"""The order of a cloud's points (cells by z, then y, then x) from both ways of finding it: a bit per cell
of the points' box, and, for boxes of more than 4096 cells a point, the sort.  Points at cells drawn
without repetition come back as the sorted list of them, with their own position, colour and support,
also where min_support leaves some out."""
import numpy as np
import pytest

from helpers import arc_workload
from luvas3d.cloud import PointAccumulator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,extent", [
    (1, 1), (2, 2 ** 20 - 1), (300, 60), (300, 106), (300, 108), (2049, 255), (5000, 2 ** 19), (40000, 400), (40000, 700)])
def test_points_come_back_in_cell_order(n, extent):
    rng = np.random.default_rng(n + extent)
    at = np.unique(rng.integers(-(extent // 2), extent - extent // 2, size=(2 * n + 8, 3)), axis=0)
    at = at[rng.permutation(len(at))[:n]]
    cell = 0.25
    s = np.zeros((len(at), 9))
    s[:, :3] = (at + 0.5) * cell
    s[:, 5] = 1.0
    s[:, 6:] = np.abs(at) % 251
    twice = rng.random(len(at)) < 0.5
    acc = PointAccumulator(cell)
    acc.add_points(s)
    acc.add_points(s[twice])
    for least in (1, 2):
        keep = twice if least == 2 else np.ones(len(at), bool)
        c = acc.cloud(min_support=least)
        want = at[keep]
        order = np.lexsort((want[:, 0], want[:, 1], want[:, 2]))
        np.testing.assert_array_equal(c.cells, want[order])
        np.testing.assert_array_equal(c.positions, s[keep][order, :3].astype(np.float32))
        np.testing.assert_array_equal(c.colors, (np.abs(want[order]) % 251).astype(np.uint8))
        np.testing.assert_array_equal(c.support, np.where(twice[keep][order], 2, 1))


@pytest.mark.parametrize("size", [(1, 1), (7, 3), (33, 9), (64, 16)])
def test_add_map_counts_every_pixel(size):
    """Partial tiles of the map on both edges: every valid pixel is a sample, in the cell of its own
    world point."""
    from luvas3d import packing

    W, H = size
    views, _, _, _ = arc_workload(n=1, W=W, H=H, f=1.2 * max(W, H))
    rng = np.random.default_rng(W * 100 + H)
    depth = rng.uniform(1.0, 3.0, (H, W)).astype(np.float16)
    packed = depth.view(np.uint16).astype(np.uint32) | (rng.integers(0, 4096, (H, W), dtype=np.uint32) << 16)
    packed[rng.random((H, W)) < 0.1] = 0
    acc = PointAccumulator(0.05)
    acc.add_depth_map(views[0], np.full((2, 2, 3), 9, np.uint8), packed=packed)
    c = acc.cloud()
    valid, d, _ = packing.unpack_samples(packed)
    k, R, t = views[0].intrinsics, np.asarray(views[0].pose.R), np.asarray(views[0].pose.t)
    y, x = np.nonzero(valid)
    cam = np.stack([(x - k.cx) / k.fx * d[valid], (y - k.cy) / k.fy * d[valid], d[valid]], -1)
    cells, count = np.unique(np.floor((cam - t) @ R / 0.05).astype(int), axis=0, return_counts=True)
    order = np.lexsort((cells[:, 0], cells[:, 1], cells[:, 2]))
    np.testing.assert_array_equal(c.cells, cells[order])
    np.testing.assert_array_equal(c.support, count[order])
    assert (c.colors == 9).all()
