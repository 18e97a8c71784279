"""The passes that cut chunk records into steps take the records' size from
the cull that wrote them, also where that cull is replayed from a capture and
the pass is not: pools of 149 and 148 batches on 148 SMs have records of
different sizes."""
import numpy as np
import pytest

from scenes import blob_cloud
from test_gpu_render import camera, make_cloud

pytestmark = pytest.mark.gpu

STAGE_DEPTH, STAGE_COLOR, STAGE_RESOLVE = 1, 2, 4


@pytest.fixture(scope="module")
def ctx(cr):
    return cr.Context(0)


def scene(cr, orc, ctx, **kw):
    torch = pytest.importorskip("torch")
    cloud, _ = make_cloud(cr, orc, ctx, *blob_cloud(149 * 10240, 6))
    assert cloud.residentBatchCount == 149
    w, h = 97, 61
    ras = cr.ComputeRasteriser(ctx)
    # Every point of a covered pixel counts, however far behind.
    ras.configuration = cr.ComputeRasteriserConfiguration(enableCLOD=False, depthTolerance=1.0,
                                                          **kw)
    ras.addPointCloud(cloud)
    ras.resize((w, h))
    ras.update(camera(cr, (0.2, 0.1, 1.6), w=w, h=h))
    return torch, cloud, ras, w, h


def captured(torch, ctx, call):
    """A function that replays `call` on the context's stream."""
    call()
    ctx.synchronize()
    stream, graph = torch.cuda.ExternalStream(ctx.stream()), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        call()

    def replay():
        with torch.cuda.stream(stream):
            graph.replay()
    return replay


def test_colour_stage_after_a_replayed_depth_stage(cr, orc, ctx):
    torch, cloud, ras, w, h = scene(cr, orc, ctx, applyTint=True)
    cloud.tintBuffer()  # zeros: the colours as they are
    replay = captured(torch, ctx, lambda: ras.encodeStages(STAGE_DEPTH))
    cloud.removeBatches([3])
    ras.encode()
    want = ras.pixels()
    assert int(want["count"].sum()) > 148 * 10240 // 4
    replay()
    ras.encodeStages(STAGE_COLOR | STAGE_RESOLVE)
    assert np.array_equal(ras.pixels(), want)


def test_adjoint_after_a_replayed_forward(cr, orc, ctx):
    """A point's gradient is a sum over its one pixel: equal bits."""
    torch, cloud, ras, w, h = scene(cr, orc, ctx)
    n = cloud.capacity.maxResidentPoints
    col = cr.DeviceBuffer(ctx, n * 12, (n, 3), np.float32)
    col.upload(np.ones((n, 3), np.float32))
    img = cr.DeviceBuffer(ctx, w * h * 12, (h, w, 3), np.float32)
    ones = cr.DeviceBuffer(ctx, w * h * 12, (h, w, 3), np.float32)
    ones.upload(np.ones((h, w, 3), np.float32))
    grad = cr.DeviceBuffer(ctx, n * 12, (n, 3), np.float32)

    def adjoint():
        grad.upload(np.zeros((n, 3), np.float32))
        ras.backwardColors(cloud, ones, grad)
        return grad.download()

    replay = captured(torch, ctx, lambda: ras.forwardF32(cloud, col, img))
    cloud.removeBatches([3])
    ras.forwardF32(cloud, col, img)
    want = adjoint()
    assert (want > 0).any(1).sum() > 148 * 10240 // 4
    replay()
    assert np.array_equal(adjoint(), want)


@pytest.mark.parametrize("chunk", [256, 300, 2048])
@pytest.mark.parametrize("ppb", [1, 3, 31, 33, 64, 255, 257, 1025, 2051])
def test_fragments_of_batches_that_start_unaligned(cr, orc, ctx, ppb, chunk):
    """One-view and batched frames of single pixels, whose fragments each warp
    packs for the same warp of the colour pass: bit for bit against the oracle."""
    from test_gpu_render import assert_same, render_both
    cloud, _ = make_cloud(cr, orc, ctx, *blob_cloud(700 if ppb < 4 else 9000, 12), ppb=ppb)
    w, h = 97, 61
    cam = camera(cr, (0.2, 0.1, 1.6), w=w, h=h)
    cfg = cr.ComputeRasteriserConfiguration(depthTolerance=0.3)
    before = ctx.tuning()["chunkPoints"]
    try:
        ctx.set_tuning(chunkPoints=chunk)
        _, gpu, ref = render_both(cr, orc, ctx, [cloud], cfg, cam, w, h)
        assert_same(cr, cfg, gpu, ref)
        mv = cr.MultiViewRasteriser(ctx, [(w, h)] * 2)
        mv.configuration = cfg
        mv.addPointCloud(cloud)
        mv.render([cam, cam])
        for v in (0, 1):
            px = mv.pixels(v)
            assert np.array_equal(px["depth"], ref.depth)
            assert np.array_equal(np.stack([px[k] for k in ("red", "green", "blue", "count")], -1),
                                  ref.accum)
        mv.close()
    finally:
        ctx.set_tuning(chunkPoints=before)


@pytest.mark.parametrize("ppb", [1, 4, 16, 255, 256, 257, 260])
@pytest.mark.parametrize("tiles", [False, True])
def test_nearest_frames_of_small_records(cr, orc, ctx, ppb, tiles):
    """Records of as many points as a CTA has threads, fewer and more."""
    from test_gpu_render import assert_same, render_both
    cloud, _ = make_cloud(cr, orc, ctx, *blob_cloud(700 if ppb < 4 else 6000, 13), ppb=ppb)
    try:
        ctx.set_tuning(useTiles=tiles)
        for w, h in ((97, 61), (16, 9)):
            cfg = cr.ComputeRasteriserConfiguration(mode=cr.MODE_NEAREST)
            _, gpu, ref = render_both(cr, orc, ctx, [cloud], cfg,
                                      camera(cr, (0.2, 0.1, 1.6), w=w, h=h), w, h)
            assert_same(cr, cfg, gpu, ref)
    finally:
        ctx.set_tuning(useTiles=True)
