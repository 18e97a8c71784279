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


@pytest.mark.parametrize("chunk", [256, 300, 2048])
@pytest.mark.parametrize("ppb", [255, 257, 511, 512, 513, 10240])
def test_training_passes_at_step_edges(cr, orc, ctx, chunk, ppb):
    """The FP32 passes over batches and chunk records around their 512-point
    steps, with a chunk size set between the forward and the adjoint: the
    image is the mean of the visible points' colours and the gradient of an
    image gradient of ones is 1 / count per visible pixel.  Every visible
    point and pixel comes from the oracle's depth plane and counts; the sums
    of at most a few hundred FP32 terms in [0, 1] are held to 1e-4."""
    pos, rgba = blob_cloud(5000, 21)
    cloud, _ = make_cloud(cr, orc, ctx, pos, rgba, ppb=ppb)
    n = cloud.capacity.maxResidentPoints
    w, h = 61, 47
    cam = camera(cr, (0.2, 0.1, 1.6), w=w, h=h)
    cfg = cr.ComputeRasteriserConfiguration(enableCLOD=False)
    before = ctx.tuning()["chunkPoints"]
    try:
        ctx.set_tuning(chunkPoints=chunk)
        ras, gpu, ref = render_both(cr, orc, ctx, [cloud], cfg, cam, w, h)
        assert_same(cr, cfg, gpu, ref)
        # Colours (1, 1/2, 0): the covered pixels are exactly that.
        col = cr.DeviceBuffer(ctx, n * 12, (n, 3), np.float32)
        col.upload(np.tile(np.array([1.0, 0.5, 0.0], np.float32), (n, 1)))
        img = cr.DeviceBuffer(ctx, w * h * 12, (h, w, 3), np.float32)
        ones = cr.DeviceBuffer(ctx, w * h * 12, (h, w, 3), np.float32)
        ones.upload(np.ones((h, w, 3), np.float32))
        grad = cr.DeviceBuffer(ctx, n * 12, (n, 3), np.float32)
        grad.upload(np.zeros((n, 3), np.float32))
        ras.forwardF32(cloud, col, img)
        ctx.set_tuning(chunkPoints=4096)
        ras.backwardColors(cloud, ones, grad)
        covered = ref.accum[..., 3] > 0
        want = np.where(covered[..., None], np.array([1.0, 0.5, 0.0], np.float32), 0.0)
        assert np.abs(img.download() - want).max() <= 1e-4
        # Every covered pixel hands out 1 in all: the sum of the gradients.
        total = grad.download().astype(np.float64).sum(0)
        assert np.abs(total - covered.sum()).max() <= 1e-4 * covered.sum()
    finally:
        ctx.set_tuning(chunkPoints=before)


@pytest.mark.parametrize("ppb", [1, 333, 1024, 2050, 10240])
@pytest.mark.parametrize("mode,scale,most", [(0, 6.0, 40.0), (1, 0.004, 3.0), (1, 0.02, 9.0),
                                             (1, 0.3, 64.0)])
def test_splats(cr, orc, ctx, ppb, mode, scale, most):
    """Footprints from a pixel to the largest (radius 16), with batches that
    start unaligned, at a frame edge, with and without tiles."""
    pos, rgba = blob_cloud(300 if ppb == 1 else 5000, 33)
    cloud, _ = make_cloud(cr, orc, ctx, pos, rgba, ppb=ppb)
    cfg = cr.ComputeRasteriserConfiguration(pointSizeMode=mode, pointSizeScale=scale,
                                            maximumPointSize=most, depthTolerance=0.02)
    try:
        for tiles in (True, False):
            ctx.set_tuning(useTiles=tiles)
            for w, h in ((211, 97), (19, 23)):
                cam = camera(cr, (0.3, 0.1, 1.2), w=w, h=h)
                _, gpu, ref = render_both(cr, orc, ctx, [cloud], cfg, cam, w, h)
                assert_same(cr, cfg, gpu, ref)
    finally:
        ctx.set_tuning(useTiles=True)


@pytest.mark.parametrize("chunk", [256, 1000, 1025, 5000])
def test_splats_of_two_clouds_and_chunk_sizes(cr, orc, ctx, chunk):
    a, _ = make_cloud(cr, orc, ctx, *blob_cloud(7000, 41), ppb=2051)
    b, _ = make_cloud(cr, orc, ctx, *lattice_cloud(16, 42), ppb=1500)
    cfg = cr.ComputeRasteriserConfiguration(pointSizeMode=1, pointSizeScale=0.01,
                                            maximumPointSize=7.0, holeFillIterations=3,
                                            colorizeChunks=chunk == 1000)
    before = ctx.tuning()["chunkPoints"]
    try:
        ctx.set_tuning(chunkPoints=chunk)
        w, h = 240, 130
        _, gpu, ref = render_both(cr, orc, ctx, [a, b], cfg, camera(cr, (0.5, 0.2, 2.2), w=w, h=h),
                                  w, h)
        assert_same(cr, cfg, gpu, ref)
    finally:
        ctx.set_tuning(chunkPoints=before)


def test_splats_past_the_packed_bound(cr, ctx):
    """More samples in a splat's pixels than the packed adds can hold: the
    frame is drawn again with 32-bit adds, every sum modulo 2^32."""
    from test_gpu_accum_wrap import LIMIT, stacked_cloud
    samples, w = LIMIT + 11, 16
    cloud = stacked_cloud(cr, ctx, samples)
    ras = cr.ComputeRasteriser(ctx)
    ras.configuration = cr.ComputeRasteriserConfiguration(
        enableCLOD=False, enableLODDither=False, pointSizeMode=0, pointSizeScale=9.0,
        maximumPointSize=3.0)  # 9 / 3 units away: 3 pixels, radius 1
    ras.addPointCloud(cloud)
    ras.resize((w, w))
    ras.update(camera(cr, (0.0, 0.0, 3.0), w=w, h=w))
    ras.encode()
    px = ras.pixels()
    hit = np.argwhere(px["count"] != 0)
    assert len(hit) == 9 and (hit.max(0) - hit.min(0)).tolist() == [2, 2]
    s = (255 * samples) % (1 << 32)
    for y, x in hit:
        assert [int(px[y, x][k]) for k in ("red", "green", "blue", "count")] == [s, s, s, samples]
    rgba = ras.outputRGBA8()
    assert (rgba[hit[:, 0], hit[:, 1], 3] == 255).all()


@pytest.mark.parametrize("ppb,files", [(255, 1), (257, 5), (10240, 4)])
@pytest.mark.parametrize("most", [1.0, 5.0])
def test_effects_at_step_edges(cr, orc, ctx, ppb, files, most):
    """Displacement and tint over batches around the 256-point steps, with a
    file table in the kernel parameters and one past them, and with single
    pixels and splats.  With no displacement and a tint of weight zero the
    frame is the plain one's; with a weight below zero nothing is coloured."""
    from scenes import to_product_packed
    pos, rgba = blob_cloud(4000, 61)
    packed = orc.pack(pos, colors_rgba8=rgba, pointsPerBatch=ppb)
    prod = to_product_packed(cr, packed)
    prod.files = cr.identity_files(files)
    prod.batches = prod.batches.copy()
    prod.batches["fileIndex"] = np.arange(len(prod.batches)) % files
    cloud = cr.ComputeRasteriserPointCloud(ctx, packed=prod)
    w, h = 97, 61
    cam = camera(cr, (0.2, 0.1, 1.4), w=w, h=h)
    cfg = cr.ComputeRasteriserConfiguration(pointSizeMode=0, pointSizeScale=4.0,
                                            maximumPointSize=most)
    ras, gpu, ref = render_both(cr, orc, ctx, [cloud], cfg, cam, w, h)
    assert_same(cr, cfg, gpu, ref)
    cfg.applyDisplacement = cfg.applyTint = True
    cloud.displacementBuffer()
    tint = cloud.tintBuffer()
    zero = np.zeros(tint.shape, np.float32)
    for weight in (0.0, -1.0):
        zero[:, 3] = weight
        tint.upload(zero)
        ras.update(cam)
        ras.encode()
        px = ras.pixels()
        assert np.array_equal(px["depth"], ref.depth)
        accum = np.stack([px["red"], px["green"], px["blue"], px["count"]], -1)
        assert np.array_equal(accum, ref.accum if weight == 0.0 else 0 * ref.accum)


@pytest.mark.parametrize("radius", [0, 1, 10, 63, 100000])
def test_pick_window(cr, orc, ctx, radius):
    """The pick is the covered pixel nearest to the cursor, the first in row
    order among equals, at any radius and at the frame's edges: the same
    search over the index plane read back."""
    pos, rgba = blob_cloud(400, 71)
    cloud, _ = make_cloud(cr, orc, ctx, pos, rgba)
    w, h = 150, 83
    cam = camera(cr, (0.2, 0.1, 1.9), w=w, h=h)
    cfg = cr.ComputeRasteriserConfiguration(mode=cr.MODE_NEAREST)
    ras, _, _ = render_both(cr, orc, ctx, [cloud], cfg, cam, w, h)
    plane = ras.nearestIndices()
    ys, xs = np.nonzero(plane != 0xffffffff)
    for nx, ny in ((0.0, 0.0), (-1.0, 1.0), (1.0, -1.0), (0.31, -0.27), (-0.9, -0.4)):
        px = min(max(int(np.float32(nx * 0.5 + 0.5) * w), 0), w - 1)
        py = min(max(h - 1 - int(np.float32(ny * 0.5 + 0.5) * h), 0), h - 1)
        d = (xs - px) ** 2 + (ys - py) ** 2
        best = np.lexsort((xs, ys, d))[0]
        want = int(plane[ys[best], xs[best]]) if d[best] <= radius * radius else None
        assert ras.pickPointIndex((nx, ny), cloud, cam, searchRadius=radius) == want


@pytest.mark.parametrize("chunk", [512, 2048, 4096])
@pytest.mark.parametrize("batches", [147, 148, 149])
def test_record_size_of_small_clouds(cr, orc, ctx, chunk, batches):
    """Frames of both modes, of single pixels and of footprints, on either side
    of the pool size at which the cull's records change theirs (148 batches of
    10,240 points on 148 SMs), next to a cloud of small batches."""
    small, _ = make_cloud(cr, orc, ctx, *blob_cloud(900, 5), ppb=40)
    cloud, _ = make_cloud(cr, orc, ctx, *blob_cloud(batches * 10240, 6))
    assert cloud.residentBatchCount == batches
    w, h = 97, 61
    cam = camera(cr, (0.2, 0.1, 1.6), w=w, h=h)
    before = ctx.tuning()["chunkPoints"]
    try:
        ctx.set_tuning(chunkPoints=chunk)
        for mode, most in ((cr.MODE_HQS, 1.0), (cr.MODE_HQS, 3.0), (cr.MODE_NEAREST, 1.0)):
            cfg = cr.ComputeRasteriserConfiguration(mode=mode, enableCLOD=False,
                                                    maximumPointSize=most)
            _, gpu, ref = render_both(cr, orc, ctx, [small, cloud], cfg, cam, w, h)
            assert_same(cr, cfg, gpu, ref)
    finally:
        ctx.set_tuning(chunkPoints=before)
