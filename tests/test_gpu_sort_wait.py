"""The packer's sort when its bounded wait gives up: with a limit of 0 polls
every tile after a segment's first gives up at once, nothing waits, and the
order is no permutation.  The kernels behind the sort stay inside their
arrays, the next synchronising call reports CR_ERR_TIMEOUT, and the next pack
is the CPU's again."""
import numpy as np
import pytest

import white_box
from scenes import blob_cloud
from test_gpu_pack import check_region, gpu_pack

pytestmark = pytest.mark.gpu

CR_ERR_TIMEOUT = 6


@pytest.fixture(scope="module")
def inside(cr, tmp_path_factory):
    return white_box.build(str(tmp_path_factory.mktemp("white_box")), cr)


def pack_without_waiting(cr, ctx, inside, pos, rgba, bits):
    """A pack whose tiles give up, after the values' buffers were filled with
    the largest word; raises the report."""
    for k in (0, 1):
        p = cr.DeviceView(ctx, inside.sort_indices(ctx.handle, k), (len(pos),), np.uint32)
        p.upload(np.full(len(pos), 0xffffffff, np.uint32))
    limit = inside.get_sort_wait_limit(ctx.handle)
    assert limit == 1 << 22
    try:
        inside.set_sort_wait_limit(ctx.handle, 0)
        gpu_pack(cr, ctx, pos, rgba=rgba, bits=bits)
        with pytest.raises(cr.CRError) as err:
            ctx.synchronize()
        assert err.value.status == CR_ERR_TIMEOUT
        assert "sort" in str(err.value)
        ctx.synchronize()  # reported once
    finally:
        inside.set_sort_wait_limit(ctx.handle, limit)


@pytest.mark.parametrize("bits", [10, 21])
def test_pack_after_a_sort_that_gave_up(cr, orc, inside, bits):
    ctx = cr.Context(0)
    pos, rgba = blob_cloud(50000, 3)
    ref = orc.pack(pos, colors_rgba8=rgba, pointsPerBatch=10240, morton_bits=bits)
    for _ in range(2):
        cloud, src = gpu_pack(cr, ctx, pos, rgba=rgba, bits=bits)
        check_region(cloud, ref, 0, 10240, src)
        pack_without_waiting(cr, ctx, inside, pos, rgba, bits)
    cloud, src = gpu_pack(cr, ctx, pos, rgba=rgba, bits=bits)
    check_region(cloud, ref, 0, 10240, src)


def test_packs_after_a_sort_with_ties_gave_up(cr, orc, inside):
    """63-bit keys of a cloud large enough to leave out low digits: with the
    order wrong, no run of keys is walked along, and every voxel of the LOD
    grids that was claimed is set free again, so later packs of the context
    (of the same grids, and of smaller ones in the same memory) have the
    CPU's levels."""
    ctx = cr.Context(0)
    rng = np.random.default_rng(9)
    n = (1 << 19) + 4099
    pos = rng.uniform(-1.0, 1.0, (n, 3)).astype(np.float32)
    rgba = rng.integers(0, 1 << 32, n, dtype=np.uint32)
    ref = orc.pack(pos, colors_rgba8=rgba, pointsPerBatch=10240, morton_bits=21, threads=8)
    few, few_rgba = blob_cloud(30000, 4)
    few_ref = orc.pack(few, colors_rgba8=few_rgba, pointsPerBatch=10240)
    cloud, src = gpu_pack(cr, ctx, pos, rgba=rgba, bits=21)
    check_region(cloud, ref, 0, 10240, src)
    for _ in range(2):
        pack_without_waiting(cr, ctx, inside, pos, rgba, 21)
        cloud, src = gpu_pack(cr, ctx, few, rgba=few_rgba)
        check_region(cloud, few_ref, 0, 10240, src)
        cloud, src = gpu_pack(cr, ctx, pos, rgba=rgba, bits=21)
        check_region(cloud, ref, 0, 10240, src)
