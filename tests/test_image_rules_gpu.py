"""Image preparation on both sides of its rules on sizes (csrc/image.cu): how many lanes share a block of
gray bytes, and up to which target the area filter runs in one pass; bit for bit against the oracle."""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")

from luvas3d import image as I  # noqa: E402

pytestmark = pytest.mark.gpu


# 65536 targets: one lane; one row fewer: two; 100 x 100: eight of sixteen; 40 x 30: all 32
@pytest.mark.parametrize("src,dst", [((2048, 2048), (256, 256)), ((2040, 2048), (255, 256)), ((1600, 1600), (100, 100)),
                                     ((960, 1280), (30, 40)), ((1500, 4104), (500, 513))])
def test_gray_blocks(src, dst):
    g = np.random.default_rng(8).integers(0, 256, size=src, dtype=np.uint8)
    got = I.downsample_gray(torch.from_numpy(g).cuda(), dst[1], dst[0]).cpu().numpy()
    np.testing.assert_array_equal(got, oracle.downsample_gray(g, dst[1], dst[0]))


# 1.5 and 2 million targets, and a row more
@pytest.mark.parametrize("dst", [(1250, 1200), (1251, 1200), (1600, 1250), (1601, 1250)])
def test_area_filter(dst):
    a = np.random.default_rng(9).integers(0, 256, size=(1100, 1031, 4), dtype=np.uint8)
    g = np.ascontiguousarray(a[..., 2])
    np.testing.assert_array_equal(I.downsample_gray(torch.from_numpy(g).cuda(), dst[1], dst[0]).cpu().numpy(),
                                  oracle.downsample_gray(g, dst[1], dst[0]))
    np.testing.assert_array_equal(I.rgba_to_gray(torch.from_numpy(a).cuda(), dst[1], dst[0]).cpu().numpy(),
                                  oracle.rgba_to_gray(a, dst[1], dst[0]))
