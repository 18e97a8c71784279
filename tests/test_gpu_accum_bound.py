"""Packed colour adds need a bound on the samples of a pixel: it covers what
the device draws, not what the host has left.  Batches of one white point at
the origin, so a few pixels receive every sample; sums modulo 2^32."""
import numpy as np
import pytest

from test_gpu_accum_wrap import H, LIMIT, PPB, W, stacked_cloud

pytestmark = pytest.mark.gpu

DRAWN = 2000 * PPB  # above LIMIT
KEPT = 1600 * PPB   # below it
assert KEPT <= LIMIT < DRAWN


@pytest.fixture(scope="module")
def ctx(cr):
    return cr.Context(0)


def rasteriser(cr, ctx, cloud, what):
    cfg = cr.ComputeRasteriserConfiguration(enableCLOD=False, enableLODDither=False)
    if what == "splats":  # 9 / 3 units away: 3 pixels, nine in all
        cfg.pointSizeMode, cfg.pointSizeScale, cfg.maximumPointSize = 0, 9.0, 3.0
    if what == "effects":  # a tint of weight zero: the colours as they are
        cfg.applyTint = True
        cloud.tintBuffer()
    cam = cr.PerspectiveCamera(position=(0.0, 0.0, 3.0), near=0.01, far=100.0, fov=60.0,
                               aspect=1.0)
    cam.lookAt((0.0, 0.0, 0.0))
    ras = cr.ComputeRasteriser(ctx)
    ras.configuration = cfg
    ras.addPointCloud(cloud)
    ras.resize((W, H))
    ras.update(cam)
    return ras


def check(ras, what, samples):
    px = ras.pixels()
    hit = np.argwhere(px["count"] != 0)
    assert len(hit) == (9 if what == "splats" else 1)
    s = (255 * samples) % (1 << 32)
    for y, x in hit:
        assert [int(px[y, x][k]) for k in ("red", "green", "blue", "count")] == [s, s, s, samples]


@pytest.mark.parametrize("what", ["pixels", "splats", "effects"])
def test_removal_not_yet_committed(cr, ctx, what):
    """The device draws removed batches until the removal is committed."""
    cloud = stacked_cloud(cr, ctx, DRAWN)
    ras = rasteriser(cr, ctx, cloud, what)
    cloud.removeBatches(list(range(400)), commit=False)
    assert cloud.residentBatchCount == 1600
    ras.encode()
    check(ras, what, DRAWN)
    cloud.commitBatchUpdates()
    ras.encode()
    check(ras, what, KEPT)


@pytest.mark.parametrize("what", ["pixels", "splats", "effects"])
def test_captured_frame_after_batches_were_added(cr, ctx, what):
    """A captured frame draws the records that there are when it is replayed."""
    torch = pytest.importorskip("torch")
    cloud = stacked_cloud(cr, ctx, DRAWN)
    cloud.removeBatches(list(range(400)))
    ras = rasteriser(cr, ctx, cloud, what)
    ras.encode()
    check(ras, what, KEPT)
    stream, graph = torch.cuda.ExternalStream(ctx.stream()), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        ras.encode()
    with torch.cuda.stream(stream):
        graph.replay()
    check(ras, what, KEPT)
    b = np.zeros(400, cr.BATCH_DTYPE)
    b["state"], b["numPoints"] = 1, PPB
    zeros = np.zeros(PPB, np.uint32)
    cloud.addBatches(zeros, zeros, zeros, np.full(PPB, 0xFFFFFFFF, np.uint32),
                     np.zeros(PPB, np.uint8), b)
    with torch.cuda.stream(stream):
        graph.replay()
    check(ras, what, DRAWN)
