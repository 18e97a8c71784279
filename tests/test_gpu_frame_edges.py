"""Frames at the edges of the pass kernels' tiles and tables, bit for bit
against the CPU oracle (whole numbers and bytes: nothing is allowed for)."""
import numpy as np
import pytest

from scenes import blob_cloud, lattice_cloud
from test_gpu_render import assert_same, camera, make_cloud, render_both

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(cr):
    return cr.Context(0)


@pytest.mark.parametrize("w,h", [(16, 9), (37, 27), (64, 64), (333, 251)])
def test_colour_table_conflicts(cr, orc, ctx, w, h):
    """A chunk's pixels against the colour pass's table: fewer than its slots,
    a window whose pixels all have slots of their own, one whose do not, and
    far more pixels than slots."""
    pos, rgba = blob_cloud(6000, 11, scale=1.5)
    cloud, _ = make_cloud(cr, orc, ctx, pos, rgba)
    cfg = cr.ComputeRasteriserConfiguration(depthTolerance=0.5, enableCLOD=False)
    _, gpu, ref = render_both(cr, orc, ctx, [cloud], cfg, camera(cr, (0.2, 0.1, 1.6), w=w, h=h),
                              w, h)
    assert_same(cr, cfg, gpu, ref)


@pytest.mark.parametrize("w,h", [(1, 1), (3, 3), (5, 2), (67, 45), (320, 180)])
def test_nearest_frames_one_after_the_other(cr, orc, ctx, w, h):
    """Every nearest frame starts from a cleared key plane, at odd and even
    pixel counts; the pick's pass too."""
    pos, rgba = lattice_cloud(14, 5)
    cloud, _ = make_cloud(cr, orc, ctx, pos, rgba)
    cfg = cr.ComputeRasteriserConfiguration(mode=cr.MODE_NEAREST)
    for at in ((0.1, 0.2, 2.5), (2.5, 0.1, 0.4), (0.0, 0.3, 30.0)):
        ras, gpu, ref = render_both(cr, orc, ctx, [cloud], cfg, camera(cr, at, w=w, h=h), w, h)
        assert_same(cr, cfg, gpu, ref)
        ras.pickPointIndex((0.0, 0.0), cloud, camera(cr, (1.0, 1.0, 3.0), w=w, h=h))
        ras.update(camera(cr, at, w=w, h=h))
        ras.encode()
        assert np.array_equal(ras.nearestIndices(), gpu["ni"])
