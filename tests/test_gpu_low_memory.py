"""Calls that run out of device memory: they fail with an error, and the same
call works once memory is there."""
import numpy as np
import pytest

from scenes import blob_cloud
from test_gpu_pack import check_region
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


@pytest.mark.parametrize("host", [False, True])
def test_chunks_beside_a_full_gpu(cr, orc, host):
    """Thirteen nodes whose LOD grids (78 MB each at the default divisions)
    fit one at a time, not together: packed, each as the CPU packs it."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(17)
    nodes = []
    for k in range(13):
        n = 2000 + 37 * k
        nodes.append((rng.uniform(-1.0, 1.0, (n, 3)).astype(np.float32),
                      rng.integers(0, 1 << 32, n, dtype=np.uint32)))
    given = nodes
    if not host:
        given = [(torch.from_numpy(p).cuda(), torch.from_numpy(c.view("int32")).cuda())
                 for p, c in nodes]
        torch.cuda.synchronize()
    warm = cr.Context(0)  # loads the kernels; its scratch goes with it
    spare = cr.ComputeRasteriserPointCloud(warm, cr.ComputeRasteriserCapacity(6, 1000))
    for some in (given[:2], given[:1]):
        spare.addRawChunksGPU(cr.GPUPacker(warm, coarseVoxelDivisions=4), some)
    spare.close()
    warm.close()
    ctx = cr.Context(0)
    cloud = cr.ComputeRasteriserPointCloud(ctx, cr.ComputeRasteriserCapacity(3 * 13, 1000))
    with LeaveFree(cr, ctx, 200 * MB):
        first = cloud.addRawChunksGPU(cr.GPUPacker(ctx), given)
        assert len(first) == 13
        for f, (pos, rgba) in zip(first, nodes):
            ref = orc.pack(pos, colors_rgba8=rgba, pointsPerBatch=1000)
            check_region(cloud, ref, f, 1000)
    # With memory back the nodes go together.
    cloud.clearAllBatches()
    assert cloud.addRawChunksGPU(cr.GPUPacker(ctx), given) == first
    for f, (pos, rgba) in zip(first, nodes):
        ref = orc.pack(pos, colors_rgba8=rgba, pointsPerBatch=1000)
        check_region(cloud, ref, f, 1000)
