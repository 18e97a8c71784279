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
