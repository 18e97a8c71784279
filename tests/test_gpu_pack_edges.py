"""The packer's kernels at the edges of their tiles, bit for bit against the
CPU oracle's pack: whole numbers and bytes, so nothing is allowed for."""
import numpy as np
import pytest

from scenes import blob_cloud
from test_gpu_pack import check_region, gpu_pack

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(cr):
    return cr.Context(0)


@pytest.mark.parametrize("n,ppb", [(1, 1), (33, 1), (513, 512), (1000, 31), (4096, 4097),
                                   (70001, 65535)])
@pytest.mark.parametrize("lod", [1, 4, 5])
def test_batch_sizes_and_levels(cr, orc, ctx, n, ppb, lod):
    """Batches of one point to the largest, with the four-level kernel's last
    level count and the eight-level kernel's first."""
    pos, rgba = blob_cloud(n, n + lod, scale=2.0)
    ref = orc.pack(pos, colors_rgba8=rgba, pointsPerBatch=ppb, lodLevels=lod,
                   coarseVoxelDivisions=5)
    cloud, src = gpu_pack(cr, ctx, pos, rgba=rgba, ppb=ppb, lod=lod, divs=5)
    check_region(cloud, ref, 0, ppb, src)


@pytest.mark.parametrize("bits", [10, 21])
@pytest.mark.parametrize("device", [False, True])
def test_many_chunks_in_one_call(cr, orc, ctx, bits, device):
    """Chunks around the tile and block sizes, one of a single point, one
    whose points all coincide (no sort pass moves anything) and one of a
    plane, packed by shared launches: each as the CPU packs it alone."""
    torch = pytest.importorskip("torch")
    ppb = 1000
    chunks = []
    for k, n in enumerate((1, 255, 4096, 4097, 9000, 300, 12288)):
        pos, rgba = blob_cloud(n, 40 + k, scale=0.5 + k)
        if k == 4:
            pos[:] = pos[0]
        if k == 5:
            pos[:, 2] = 0.25
        chunks.append((pos, rgba))
    cloud = cr.ComputeRasteriserPointCloud(ctx, cr.ComputeRasteriserCapacity(40, ppb))
    given = chunks
    if device:
        given = [(torch.from_numpy(p).cuda(), torch.from_numpy(c.view("int32")).cuda())
                 for p, c in chunks]
        torch.cuda.synchronize()
    first = cloud.addRawChunksGPU(cr.GPUPacker(ctx, mortonBits=bits), given)
    assert len(first) == len(chunks)
    for f, (pos, rgba) in zip(first, chunks):
        ref = orc.pack(pos, colors_rgba8=rgba, pointsPerBatch=ppb, morton_bits=bits)
        check_region(cloud, ref, f, ppb)
    assert cloud.pointCount == sum(len(p) for p, _ in chunks)


def test_refused_chunk_is_still_refused(cr, ctx):
    """A chunk with an infinite coordinate has no LOD grid: the call fails and
    nothing of it becomes resident, as before."""
    pos, rgba = blob_cloud(500, 3)
    bad = pos.copy()
    bad[7, 1] = float("inf")
    cloud = cr.ComputeRasteriserPointCloud(ctx, cr.ComputeRasteriserCapacity(8, 256))
    with pytest.raises(cr.CRError):
        cloud.addRawChunksGPU(cr.GPUPacker(ctx), [(pos, rgba), (bad, rgba)])
    assert cloud.residentBatchCount == 0


def test_voxel_grids_between_runs(cr, orc):
    """The LOD grids are cleared by the runs themselves: packs of one level, of
    a single voxel, of coarse and fine grids and of chunks, one after the other
    in one context, each as the CPU packs it."""
    ctx = cr.Context(0)
    runs = [(700, 1, 64, 1.0), (1, 2, 1, 1.0), (900, 2, 1, 1.0), (5000, 4, 9, 1.0),
            (5000, 4, 64, 7.0), (300, 8, 2, 0.3), (5000, 3, 33, 2.0), (64, 4, 64, 1.0)]
    for n, lod, divs, scale in runs + runs[::-1]:
        pos, rgba = blob_cloud(n, n + lod + divs, scale=scale)
        ref = orc.pack(pos, colors_rgba8=rgba, pointsPerBatch=512, lodLevels=lod,
                       coarseVoxelDivisions=divs)
        cloud, src = gpu_pack(cr, ctx, pos, rgba=rgba, ppb=512, lod=lod, divs=divs)
        check_region(cloud, ref, 0, 512, src)
        two = cr.ComputeRasteriserPointCloud(ctx, cr.ComputeRasteriserCapacity(30, 512))
        packer = cr.GPUPacker(ctx, lodLevels=lod, coarseVoxelDivisions=divs)
        for first in two.addRawChunksGPU(packer, [(pos, rgba), (pos, rgba)]):
            check_region(two, ref, first, 512)


@pytest.mark.parametrize("kind", ["spread", "ties", "crowded", "outlier"])
@pytest.mark.parametrize("n", [(1 << 19) - 1, (1 << 19) + 4099])
def test_low_digits_left_out(cr, orc, ctx, kind, n):
    """63-bit keys around the size from which the sort samples them: spread
    points (few agree above the low digits), points with runs that do (some
    coincide, some differ in the last bits only, across the gather's CTAs),
    points crowded into a few cells and a cloud shrunk by one far point (the
    sample keeps every pass): the CPU pack's order each time."""
    rng = np.random.default_rng(n + len(kind))
    pos = rng.uniform(-1.0, 1.0, (n, 3)).astype(np.float32)
    if kind == "ties":
        pos[1000:1700] = pos[999]
        pos[5000:9000:2] = pos[5001:9001:2]
        pos[20000:26000] = pos[20000] + rng.uniform(-3e-5, 3e-5, (6000, 3)).astype(np.float32)
    elif kind == "crowded":
        pos = (pos[rng.integers(0, 50, n)] +
               rng.uniform(-1e-4, 1e-4, (n, 3))).astype(np.float32)
    elif kind == "outlier":
        pos[7] = 5000.0
    rgba = rng.integers(0, 1 << 32, n, dtype=np.uint32)
    ref = orc.pack(pos, colors_rgba8=rgba, pointsPerBatch=10240, morton_bits=21, threads=8)
    cloud, src = gpu_pack(cr, ctx, pos, rgba=rgba, bits=21)
    check_region(cloud, ref, 0, 10240, src)
