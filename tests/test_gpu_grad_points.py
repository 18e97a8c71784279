"""The FP32 forward and adjoint point by point against the FP64 oracle, with a
colour of its own for every point: over batches and chunk records around the
512-point steps of the passes, and on both sides of the 64 points a pixel from
which the depth plane is drawn through screen tiles."""
import numpy as np
import pytest

from scenes import blob_cloud, oracle_cloud_from_device, oracle_config
from test_gpu_render import camera, make_cloud

pytestmark = pytest.mark.gpu

ULP = 2.0 ** -24  # half a unit in the last place of an FP32 value in [1, 2), relative


@pytest.fixture(scope="module")
def ctx(cr):
    return cr.Context(0)


@pytest.mark.parametrize("chunk", [256, 300, 2048])
@pytest.mark.parametrize("ppb", [255, 257, 511, 512, 513, 10240])
@pytest.mark.parametrize("tolerance", [0.01, 1.0])
@pytest.mark.parametrize("size", ["many", "over", "under"])
def test_every_points_colour_and_gradient(cr, orc, ctx, chunk, ppb, tolerance, size):
    """Image: the mean of K colours in [0, 1], summed in any order: at most
    (K + 2) half units.  Gradient of a point: dL / K of its one pixel, from
    dL rounded to FP32: two roundings, held to three half units; 0 exactly
    where the oracle's is."""
    pos, rgba = blob_cloud(5000, 21)
    cloud, _ = make_cloud(cr, orc, ctx, pos, rgba, ppb=ppb)
    n = cloud.capacity.maxResidentPoints
    # Frames one row high about n / 64 pixels, and an ordinary one.
    w, h = {"many": (61, 47), "over": ((n - 1) // 64, 1), "under": (-(-n // 64), 1)}[size]
    assert size == "many" or (n > 64 * w * h) == (size == "over")
    cam = camera(cr, (0.2, 0.1, 1.6), w=64, h=48)  # its aspect whatever the frame's
    cfg = cr.ComputeRasteriserConfiguration(enableCLOD=False, depthTolerance=tolerance)
    rng = np.random.default_rng(n + chunk)
    colors = rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32)
    target = rng.uniform(0.0, 1.0, (h, w, 3))
    ras = cr.ComputeRasteriser(ctx)
    ras.configuration = cfg
    ras.addPointCloud(cloud)
    ras.resize((w, h))
    ras.update(cam)
    ref = orc.render(oracle_cloud_from_device(orc, cloud), oracle_config(orc, cfg),
                     cam.viewMatrix, cam.projectionMatrix, w, h)
    count = ref.accum[..., 3].astype(np.float64)
    assert count.sum() > (4000 if tolerance == 1.0 else 50)
    ref64 = orc.hqs_grad_f64(oracle_cloud_from_device(orc, cloud), oracle_config(orc, cfg),
                             cam.viewMatrix, cam.projectionMatrix, w, h, colors, target, 0.5)

    def buf(shape, values=None):
        b = cr.DeviceBuffer(ctx, int(np.prod(shape)) * 4, shape, np.float32)
        b.upload(np.zeros(shape, np.float32) if values is None else values.astype(np.float32))
        return b

    image, grad = buf((h, w, 3)), buf((n, 3))
    before = ctx.tuning()["chunkPoints"]
    try:
        ctx.set_tuning(chunkPoints=chunk)
        ras.forwardF32(cloud, buf((n, 3), colors), image)
        ctx.set_tuning(chunkPoints=4096)
        ras.backwardColors(cloud, buf((h, w, 3), ref64["image"] - target), grad)
    finally:
        ctx.set_tuning(chunkPoints=before)
    off = np.abs(image.download().astype(np.float64) - ref64["image"])
    assert (off <= (count[..., None] + 2.0) * ULP).all()
    g, g64 = grad.download().astype(np.float64), ref64["grad"]
    assert np.count_nonzero(g64.any(1)) == int(count.sum())
    assert (np.abs(g - g64) <= 3.0 * ULP * np.abs(g64)).all()
