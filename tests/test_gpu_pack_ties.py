"""63-bit packs whose sort leaves out low digits, so that the gather orders the
runs of keys that agree above them: against the CPU oracle's pack, whole
numbers and bytes.  Whether digits were left out is read from the sort's
tie word."""
import numpy as np
import pytest

import white_box
from test_gpu_pack import check_region, gpu_pack

pytestmark = pytest.mark.gpu

CTA = 1024  # points that a CTA of the gather orders


@pytest.fixture(scope="module")
def inside(cr, tmp_path_factory):
    return white_box.build(str(tmp_path_factory.mktemp("white_box")), cr)


def runs_above(pos, low):
    """(first, length) of the runs of 63-bit Morton keys that agree above their
    low bits, in key order."""
    lo = pos.min(0)
    q = ((pos - lo) * (np.float32(2097151.0) / (pos.max(0) - lo))).clip(0, 2097151)
    q = q.astype(np.uint64)
    key = np.zeros(len(pos), np.uint64)
    for b in range(21):
        for a in range(3):
            key |= ((q[:, a] >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b + 2 - a)
    top = np.sort(key) >> np.uint64(low)
    first = np.flatnonzero(np.r_[True, top[1:] != top[:-1]])
    return first, np.diff(np.r_[first, len(top)])


def cloud_with_runs(n, seed, equal, close):
    """Uniform points; for every length in `equal` that many in one place, and
    for every length in `close` that many within 1e-5 of one."""
    rng = np.random.default_rng(seed)
    pos = rng.uniform(-1.0, 1.0, (n, 3)).astype(np.float32)
    order = rng.permutation(n)
    at = 0
    for lengths, wide in ((equal, 0.0), (close, 1e-5)):
        for r in lengths:
            k = order[at:at + r]
            pos[k] = pos[k[0]] + rng.uniform(-wide, wide, (r, 3)).astype(np.float32)
            at += r
    return pos, rng.integers(0, 1 << 32, n, dtype=np.uint32)


N = (1 << 19) + 4099


@pytest.mark.parametrize("n", [1 << 19, N])
@pytest.mark.parametrize("equal,close", [
    ((2, 2, 3, 7, 8, 9, 10, 17), (2, 3, 9, 10, 11, 16, 17, 18, 33)),
    ((700,), (690,)),
    ((31, 100, 255, 257), (64, 65, 300, 301)),
])
def test_runs_are_put_in_order(cr, orc, inside, n, equal, close):
    pos, rgba = cloud_with_runs(n, len(equal) + n, equal, close)
    first, length = runs_above(pos, 32)
    # The rule on a run's mean (6 keys) and on the longest (1,024), with room
    # for the sample's spread.
    assert (length.astype(np.float64) ** 2).sum() / n < 5.0 and length.max() < 800
    if max(equal) > 500:
        long = length > 400
        assert long.sum() == 2
        assert (first[long] // CTA != (first + length - 1)[long] // CTA).any()
    ctx = cr.Context(0)
    ref = orc.pack(pos, colors_rgba8=rgba, pointsPerBatch=10240, morton_bits=21, threads=8)
    cloud, src = gpu_pack(cr, ctx, pos, rgba=rgba, bits=21)
    ties = cr.DeviceView(ctx, inside.sort_ties(ctx.handle), (1,), np.uint32).download()
    assert ties[0] in (24, 32)
    check_region(cloud, ref, 0, 10240, src)
    # Without source indices the places are the same.
    packer = cr.GPUPacker(ctx, mortonBits=21)
    packer.pack(pos, rgba, into=cloud)
    check_region(cloud, ref, 0, 10240)


def test_a_long_run_keeps_every_digit(cr, orc, inside):
    """1,500 keys in one place leave the mean below its bound, but not the
    longest run."""
    pos, rgba = cloud_with_runs(N, 3, (1500,), ())
    _, length = runs_above(pos, 24)
    assert (length.astype(np.float64) ** 2).sum() / N < 5.6 and length.max() >= 1500
    ctx = cr.Context(0)
    ref = orc.pack(pos, colors_rgba8=rgba, pointsPerBatch=10240, morton_bits=21, threads=8)
    cloud, src = gpu_pack(cr, ctx, pos, rgba=rgba, bits=21)
    ties = cr.DeviceView(ctx, inside.sort_ties(ctx.handle), (1,), np.uint32).download()
    assert ties[0] == 0
    check_region(cloud, ref, 0, 10240, src)


@pytest.mark.parametrize("n,ppb", [(1000, 2), (5000, 127), (5000, 128), (5000, 129), (9000, 1920),
                                   (9000, 1921), (9000, 2049)])
@pytest.mark.parametrize("lod", [4, 6])
def test_batches_by_warps(cr, orc, n, ppb, lod):
    """Batches on either side of the sizes at which their kernel takes another
    warp, from one warp to all of them."""
    ctx = cr.Context(0)
    rng = np.random.default_rng(n + ppb)
    pos = rng.uniform(-1.0, 1.0, (n, 3)).astype(np.float32)
    rgba = rng.integers(0, 1 << 32, n, dtype=np.uint32)
    ref = orc.pack(pos, colors_rgba8=rgba, pointsPerBatch=ppb, lodLevels=lod,
                   coarseVoxelDivisions=3)
    cloud, src = gpu_pack(cr, ctx, pos, rgba=rgba, ppb=ppb, lod=lod, divs=3)
    check_region(cloud, ref, 0, ppb, src)


@pytest.mark.parametrize("share", [0.5, 1.0])
def test_points_in_one_place(cr, orc, inside, share):
    """Half of the cloud, or all of it, in one place: every sample meets the
    others, every claim of a level the same voxel."""
    rng = np.random.default_rng(5)
    pos = rng.uniform(-1.0, 1.0, (N, 3)).astype(np.float32)
    pos[rng.permutation(N)[:int(share * N)]] = (0.25, -0.5, 0.125)
    rgba = rng.integers(0, 1 << 32, N, dtype=np.uint32)
    ctx = cr.Context(0)
    ref = orc.pack(pos, colors_rgba8=rgba, pointsPerBatch=10240, morton_bits=21, threads=8)
    cloud, src = gpu_pack(cr, ctx, pos, rgba=rgba, bits=21)
    ties = cr.DeviceView(ctx, inside.sort_ties(ctx.handle), (1,), np.uint32).download()
    assert ties[0] == 0
    check_region(cloud, ref, 0, 10240, src)
