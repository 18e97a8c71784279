"""Calls that run out of device memory: they fail with an error, and the same
call works once memory is there."""
import numpy as np
import pytest

from scenes import blob_cloud
from test_gpu_render import assert_same, camera, make_cloud, render_both

pytestmark = pytest.mark.gpu

CR_ERR_OUT_OF_MEMORY = 2
MB = 1 << 20


@pytest.fixture(scope="module")
def ctx(cr):
    return cr.Context(0)


class LeaveFree:
    """Device memory held until about `left` bytes are free."""

    def __init__(self, cr, ctx, left: int):
        torch = pytest.importorskip("torch")
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        assert free > left, "the test needs an otherwise unused GPU"
        self.held = cr.DeviceBuffer(ctx, free - left)

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.held.close()


def test_fp32_planes_after_running_out_of_memory(cr, orc, ctx):
    """A frame's FP32 sums (256 MB) fit, their counts (64 MB) behind them do
    not: the forward is refused, and refused again, as the adjoint is; with
    memory back it draws the colours (1, 1/2, 0) where the oracle has
    samples, and nothing elsewhere (whole numbers of samples: exact to the
    rounding of at most a few hundred FP32 terms in [0, 1])."""
    pos, rgba = blob_cloud(3000, 5)
    cloud, _ = make_cloud(cr, orc, ctx, pos, rgba)
    n = cloud.capacity.maxResidentPoints
    w = h = 4096
    cfg = cr.ComputeRasteriserConfiguration(enableCLOD=False)
    # The kernels are loaded by a first, small frame.
    cam = camera(cr, (0.2, 0.1, 1.6), w=w, h=h)
    ras, gpu, ref = render_both(cr, orc, ctx, [cloud], cfg, cam, w, h)
    assert_same(cr, cfg, gpu, ref)
    col = cr.DeviceBuffer(ctx, n * 12, (n, 3), np.float32)
    col.upload(np.tile(np.array([1.0, 0.5, 0.0], np.float32), (n, 1)))
    grad = cr.DeviceBuffer(ctx, n * 12, (n, 3), np.float32)
    img = cr.DeviceBuffer(ctx, w * h * 12, (h, w, 3), np.float32)
    small = cr.ComputeRasteriser(ctx)
    small.configuration = cfg
    small.addPointCloud(cloud)
    small.resize((64, 64))
    small.update(cam)
    small.forwardF32(cloud, col, img)
    ras.update(cam)
    with LeaveFree(cr, ctx, 290 * MB):
        for _ in range(2):
            with pytest.raises(cr.CRError) as err:
                ras.forwardF32(cloud, col, img)
            assert err.value.status == CR_ERR_OUT_OF_MEMORY
            with pytest.raises(cr.CRError):
                ras.backwardColors(cloud, img, grad)
    ras.forwardF32(cloud, col, img)
    covered = ref.accum[..., 3] > 0
    assert covered.any()
    want = np.where(covered[..., None], np.array([1.0, 0.5, 0.0], np.float32), np.float32(0.0))
    assert np.abs(img.download() - want).max() <= 1e-4
