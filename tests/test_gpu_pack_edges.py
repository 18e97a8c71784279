"""The packer's kernels at the edges of their tiles, bit for bit against the
CPU oracle's pack: whole numbers and bytes, so nothing is allowed for."""
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
