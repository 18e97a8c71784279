"""What a user of the rasteriser has it do, as cases that can be timed.

A case is a dict of plain values; its "kind" says which entry points it goes
through:

  frame   ComputeRasteriser.update + encode, and the image copied to pinned
          memory while the next frame is drawn (or, "out": "planes", the
          depth plane and the accumulators taken on the device)
  views   MultiViewRasteriser.render: a set of views of one cloud
  pick    ComputeRasteriser.pickPointIndex: the point under the cursor
  pack    GPUPacker.pack: raw points to a cloud's slot pool
  chunks  ComputeRasteriserPointCloud.addRawChunksGPU: raw nodes of a stream
          into free slots of a pool
  train   forwardF32 + l2_loss + backwardColors over a set of views: one
          step on learnable colours

Clouds are the two synthetic scenes of the repository's benchmark and tests
(the 4 km heightfield and the jittered lattice), another one for each seed;
the cameras are drawn as the benchmark draws its poses.
"""
import importlib
import math

import numpy as np
import torch

cr = importlib.import_module("satin-computerasteriser_b200")

BATCH = 10240  # points per batch: the library's default
EXTENT = 4000.0  # side of the heightfield, metres


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # The smallest call: one streamed node's points in a thumbnail, where
        # launches and host calls are all there is.
        _frame("node_nearest_360p", scene="lattice", points=52 ** 3, w=640, h=360, mode="nearest"),
        # A small cloud in a window, drawn for a consumer on the GPU.
        _frame("lattice_1m_720p", scene="lattice", points=100 ** 3, w=1280, h=720, out="planes"),
        # The headline workload, both modes: a large terrain at full HD.
        _frame("terrain_100m_1080p", points=100_000_000, w=1920, h=1080),
        _frame("terrain_100m_nearest_1080p", points=100_000_000, w=1920, h=1080, mode="nearest"),
        # Without level of detail (every point of the view drawn), at an odd
        # size, with a ragged last batch, for a consumer on the GPU (the copy
        # of an image this cheap to draw would take longer than drawing it).
        _frame("terrain_20m_all_points", points=19_999_981, w=1913, h=1077, clod=False,
               out="planes"),
        # World-sized splats and hole filling: a closed surface.
        _frame("terrain_20m_splats", points=20_000_000, w=1920, h=1080, splat=0.5, fill=2),
        # The per-point effects (displacement and tint buffers).
        _frame("terrain_10m_effects", points=10_000_000, w=1920, h=1080, effects=True,
               out="planes"),
        # Many views of mixed sizes of one cloud in a call.
        {"name": "views_64_50m", "kind": "views", "points": 50_000_000, "views": 64},
        # The point under the cursor.
        {"name": "pick_20m_1080p", "kind": "pick", "points": 20_000_000, "w": 1920, "h": 1080},
        # A whole scan packed with 63-bit Morton keys from records on the GPU.
        {"name": "pack_100m_63bit", "kind": "pack", "points": 100_000_000, "bits": 21,
         "records": True},
        # The nodes of a streamed scan: separate positions and float colours,
        # ten nodes of about 140 thousand points to a call.
        {"name": "chunks_10x140k", "kind": "chunks", "points": 140_000, "chunks": 10, "bits": 10},
        # One step of fitting every point's colour to pictures.
        {"name": "train_10m_16x512", "kind": "train", "points": 10_000_000, "views": 16, "w": 512,
         "h": 512},
    ]


def _frame(name=None, scene="terrain", points=0, w=0, h=0, mode="hqs", out="image", clod=True,
           splat=0.0, fill=0, effects=False):
    c = {"kind": "frame", "scene": scene, "points": points, "w": w, "h": h, "mode": mode,
         "out": out, "clod": clod, "splat": splat, "fill": fill, "effects": effects}
    return dict(c, name=name) if name else c


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng):
    w = _log(rng, 320, 2560)
    return w, max(180, int(w * rng.choice((9 / 16, 3 / 4, 1.0, 0.5625 + rng.uniform(-0.1, 0.3)))))


def draw(rng):
    kind = rng.choice(("frame", "frame", "frame", "frame", "frame", "views", "pick", "pack",
                       "chunks", "train"))
    if kind == "frame":
        w, h = _size(rng)
        what = rng.choice(("hqs", "hqs", "hqs", "nearest", "nearest", "all", "splats", "effects"))
        most = {"hqs": 100e6, "nearest": 100e6}.get(what, 20e6)
        scene = rng.choice(("terrain", "terrain", "terrain", "lattice"))
        n = _log(rng, 5e4, 8e6) if scene == "lattice" else _log(rng, 1e5, most)
        if scene == "lattice":
            n = round(n ** (1 / 3)) ** 3
        splat = 0.0
        if what == "splats":  # metres of the terrain; the lattice is 2 wide
            splat = rng.uniform(0.3, 1.0) if scene == "terrain" else rng.uniform(0.002, 0.006)
        return _frame(scene=scene, points=n, w=w, h=h,
                      mode="nearest" if what == "nearest" else "hqs",
                      out="image" if what == "nearest" else rng.choice(("image", "image", "planes")),
                      clod=what != "all" and rng.random() < 0.9, splat=splat,
                      fill=rng.choice((0, 1, 2, 4)) if splat else rng.choice((0, 0, 0, 1)),
                      effects=what == "effects")
    if kind == "views":
        return {"kind": kind, "points": _log(rng, 1e6, 5e7), "views": rng.randint(4, 64)}
    if kind == "pick":
        w, h = _size(rng)
        return {"kind": kind, "points": _log(rng, 1e5, 5e7), "w": w, "h": h}
    if kind == "pack":
        return {"kind": kind, "points": _log(rng, 1e5, 1e8), "bits": rng.choice((10, 21)),
                "records": rng.random() < 0.5}
    if kind == "chunks":
        return {"kind": kind, "points": _log(rng, 2e4, 5e5), "chunks": rng.randint(1, 16),
                "bits": rng.choice((10, 10, 21))}
    return {"kind": kind, "points": _log(rng, 5e5, 1e7), "views": rng.randint(2, 16),
            "w": rng.randint(200, 640), "h": rng.randint(200, 512)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
_shared = []


def _context():
    """The program's one context."""
    if not _shared:
        _shared.append(cr.Context(0))
    return _shared[0]


def _records(ctx, scene, n, seed):
    if scene == "lattice":
        return cr.synth_lattice(ctx, round(n ** (1 / 3)), seed=0xC0FFEE01 + seed)
    return cr.synth_terrain(ctx, cr.TerrainParams(seed=0xC0FFEE02 + seed), n)


def _cloud(ctx, scene, n, seed):
    cloud = cr.ComputeRasteriserPointCloud(
        ctx, cr.ComputeRasteriserCapacity(-(-n // BATCH), BATCH))
    rec = _records(ctx, scene, n, seed)
    cr.GPUPacker(ctx).pack(records=rec, into=cloud)
    ctx.synchronize()
    rec.close()
    return cloud


def _camera(scene, seed, rng, w, h):
    """Over the terrain: 300 m above the ground looking 20 to 45 degrees down;
    around the lattice: two to three and a half units from its centre."""
    if scene == "lattice":
        d = rng.normal(size=3)
        cam = cr.PerspectiveCamera(position=d / np.linalg.norm(d) * rng.uniform(2.0, 3.5),
                                   near=0.01, far=100.0, fov=60.0, aspect=w / h)
        cam.lookAt((0.0, 0.0, 0.0), up=(0.0, 0.0, 1.0))
        return cam
    x, y = rng.uniform(0.15, 0.85, 2) * EXTENT
    z = cr.terrain_height(cr.TerrainParams(seed=0xC0FFEE02 + seed), x, y) + 300.0
    return _over(np.array([x, y, z]), rng, w, h)


def _over(pos, rng, w, h):
    yaw, pitch = rng.uniform(0.0, 2.0 * math.pi), math.radians(rng.uniform(-45.0, -20.0))
    d = np.array([math.cos(pitch) * math.cos(yaw), math.cos(pitch) * math.sin(yaw),
                  math.sin(pitch)])
    cam = cr.PerspectiveCamera(position=pos, near=1.0, far=10000.0, fov=60.0, aspect=w / h)
    cam.lookAt(pos + d, up=(0.0, 0.0, 1.0))
    return cam


def _on_device(ctx, ptr, shape, dtype, owner):
    """Device memory of the library's as a tensor (it keeps its owner alive)."""
    return torch.as_tensor(cr.DeviceView(ctx, ptr, shape, dtype, owner), device="cuda")


def _pool(cloud):
    a = cloud.deviceArrays()
    out = {k: _on_device(cloud.context, a[k].ptr, a[k].shape, np.int32, cloud)
           for k in ("xyzLow", "xyzMed", "xyzHigh", "colors")}
    for k in ("batches", "levels"):
        out[k] = _on_device(cloud.context, a[k].ptr, a[k].shape, np.uint8, cloud)
    return out


def prepare(case, seed):
    state = globals()["_prepare_" + case["kind"]](case, seed)
    torch.cuda.synchronize()
    return dict(state, kind=case["kind"])


def _prepare_frame(c, seed):
    ctx, rng = _context(), np.random.default_rng(seed)
    cloud = _cloud(ctx, c["scene"], c["points"], seed)
    ras = cr.ComputeRasteriser(ctx)
    ras.addPointCloud(cloud)
    cfg = cr.ComputeRasteriserConfiguration(
        mode=cr.MODE_NEAREST if c["mode"] == "nearest" else cr.MODE_HQS, enableCLOD=c["clod"],
        holeFillIterations=c["fill"])
    if c["splat"] > 0:
        cfg.pointSizeMode, cfg.pointSizeScale, cfg.maximumPointSize = 1, c["splat"], 8.0
    if c["effects"]:
        g = torch.Generator("cuda").manual_seed(seed)
        n = cloud.capacity.maxResidentPoints
        move, tint = cloud.displacementBuffer(), cloud.tintBuffer()
        ctx.synchronize()  # zeroed on the library's stream
        wide = 0.5 if c["scene"] == "terrain" else 0.002
        _on_device(ctx, move.ptr, (n, 4), np.float32, cloud).normal_(0.0, wide, generator=g)
        _on_device(ctx, tint.ptr, (n, 4), np.float32, cloud).uniform_(0.0, 0.8, generator=g)
        cfg.applyDisplacement = cfg.applyTint = True
    ras.configuration = cfg
    ras.resize((c["w"], c["h"]))
    state = {"ras": ras, "camera": _camera(c["scene"], seed, rng, c["w"], c["h"]), "turn": 0}
    if c["out"] == "planes":
        p = ras.devicePlanes()
        state["planes"] = {
            "depth": _on_device(ctx, p["depth"], (c["h"], c["w"]), np.int32, ras),
            "accum": _on_device(ctx, p["accum"], (c["h"], c["w"], 4), np.int32, ras)}
    else:
        state["images"] = [torch.empty((c["h"], c["w"], 4), dtype=torch.uint8, pin_memory=True)
                           for _ in range(2)]
    return state


def _prepare_views(c, seed):
    # A context of its own: the program draws one set of views, and the
    # library keeps that set's buffers and graphs in the context.
    ctx, rng = cr.Context(0), np.random.default_rng(seed)
    cloud = _cloud(ctx, "terrain", c["points"], seed)
    ctx.trim()
    sizes = [((256, 256), (512, 512), (1280, 720), (1920, 1080))[k]
             for k in np.random.default_rng(7).integers(0, 4, c["views"])]
    mv = cr.MultiViewRasteriser(ctx, sizes)
    mv.addPointCloud(cloud)
    images = [[torch.empty((h, w, 4), dtype=torch.uint8, pin_memory=True) for w, h in sizes]
              for _ in range(2)]
    return {"mv": mv, "cameras": [_camera("terrain", seed, rng, w, h) for w, h in sizes],
            "images": images, "turn": 0}


def _prepare_pick(c, seed):
    ctx, rng = _context(), np.random.default_rng(seed)
    cloud = _cloud(ctx, "terrain", c["points"], seed)
    ras = cr.ComputeRasteriser(ctx)
    ras.addPointCloud(cloud)
    ras.resize((c["w"], c["h"]))
    return {"ras": ras, "cloud": cloud, "camera": _camera("terrain", seed, rng, c["w"], c["h"]),
            "at": (float(rng.uniform(-0.8, 0.8)), float(rng.uniform(-0.9, 0.2)))}


def _raw(ctx, n, seed):
    """Positions (n, 3) and float colours (n, 4) of the terrain, as tensors."""
    rec = _records(ctx, "terrain", n, seed)
    ctx.synchronize()
    t = torch.as_tensor(rec, device="cuda")
    rgba = t[:, 3].contiguous().view(torch.int32)
    pos = t[:, :3].contiguous()
    col = torch.stack([((rgba >> s) & 255).float() / 255.0 for s in (0, 8, 16, 24)], 1)
    torch.cuda.synchronize()
    return pos, col


def _prepare_pack(c, seed):
    ctx, n = _context(), c["points"]
    if c["records"]:
        raw = {"records": _records(ctx, "terrain", n, seed)}
    else:
        pos, col = _raw(ctx, n, seed)
        raw = {"positions": pos, "colors": col}
    cloud = cr.ComputeRasteriserPointCloud(
        ctx, cr.ComputeRasteriserCapacity(-(-n // BATCH), BATCH))
    return {"packer": cr.GPUPacker(ctx, mortonBits=c["bits"]), "raw": raw, "cloud": cloud,
            "pool": _pool(cloud)}


def _prepare_chunks(c, seed):
    ctx = _context()
    rng = np.random.default_rng(c["points"])  # the nodes' sizes are the case's
    nodes = [_raw(ctx, max(1, int(c["points"] * rng.uniform(0.8, 1.2))), 31 * seed + k)
             for k in range(c["chunks"])]
    # A node is a patch of the terrain: a corner of it scaled down.
    nodes = [(pos * 0.05, col) for pos, col in nodes]
    slots = sum(-(-len(p) // BATCH) for p, _ in nodes)
    cloud = cr.ComputeRasteriserPointCloud(ctx, cr.ComputeRasteriserCapacity(slots, BATCH))
    return {"packer": cr.GPUPacker(ctx, mortonBits=c["bits"]), "nodes": nodes, "cloud": cloud,
            "pool": _pool(cloud)}


# --- the training cloud: packed here, so that exact() can decode it too -----
def _height(x, y, wave, phase):
    z = torch.zeros_like(x)
    for k in range(wave.shape[0]):
        z += wave[k, 2] * torch.sin(wave[k, 0] * x + wave[k, 1] * y + phase[k])
    return z


def _packed(c, seed):
    """A heightfield cut into square patches of a batch each, quantised to 30
    bits an axis: (batch minima, batch maxima, the three words) on the GPU,
    and the height function's parameters."""
    g = torch.Generator("cuda").manual_seed(seed)
    nb = -(-c["points"] // BATCH)
    side = math.ceil(math.sqrt(nb))
    k = torch.arange(nb, device="cuda")
    cell = EXTENT / side
    wave = torch.rand((6, 3), device="cuda", generator=g) - 0.5
    wave = wave * torch.tensor([0.012, 0.012, 80.0], device="cuda")
    phase = torch.rand(6, device="cuda", generator=g) * 6.2831853
    u = torch.rand((nb, BATCH, 2), device="cuda", generator=g)
    x = (u[..., 0] + (k % side)[:, None]) * cell
    y = (u[..., 1] + (k // side)[:, None]) * cell
    p = torch.stack([x, y, _height(x, y, wave, phase)], -1)
    mn, mx = p.amin(1), p.amax(1)
    q = ((p - mn[:, None]) / torch.clamp(mx - mn, min=1e-6)[:, None]).clamp(0.0, 0.99999994)
    q = (q * 1073741824.0).to(torch.int64)
    words = []
    for s in (20, 10, 0):
        v = (q >> s) & 1023
        words.append((v[..., 0] | (v[..., 1] << 10) | (v[..., 2] << 20)).to(torch.int32).reshape(-1))
    return mn, mx, words, (wave, phase)


def _train_inputs(c, seed, land):
    """Colours, target pictures and cameras of a step."""
    g = torch.Generator("cuda").manual_seed(seed + 1)
    n = -(-c["points"] // BATCH) * BATCH
    colors = torch.rand((n, 3), device="cuda", generator=g)
    targets = torch.rand((c["views"], c["h"], c["w"], 3), device="cuda", generator=g)
    rng, cams = np.random.default_rng(seed), []
    for _ in range(c["views"]):
        x, y = rng.uniform(0.15, 0.85, 2) * EXTENT
        z = float(_height(torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda"), *land))
        cams.append(_over(np.array([x, y, z + 300.0]), rng, c["w"], c["h"]))
    return colors, targets, cams


def _prepare_train(c, seed):
    ctx = _context()
    mn, mx, words, land = _packed(c, seed)
    colors, targets, cams = _train_inputs(c, seed, land)
    nb, n = mn.shape[0], mn.shape[0] * BATCH
    b = np.zeros(nb, cr.BATCH_DTYPE)
    mn, mx = mn.cpu().numpy(), mx.cpu().numpy()
    b["state"], b["numPoints"], b["firstPoint"] = 1, BATCH, np.arange(nb) * BATCH
    for k, a in enumerate("XYZ"):
        b["min" + a], b["max" + a] = mn[:, k], mx[:, k]
    cloud = cr.ComputeRasteriserPointCloud(ctx, cr.ComputeRasteriserCapacity(nb, BATCH))
    low, med, high = (w.cpu().numpy().view(np.uint32) for w in words)
    slots = cloud.addBatches(low, med, high, np.zeros(n, np.uint32), np.zeros(n, np.uint8), b)
    if slots != list(range(nb)):
        raise RuntimeError("a new pool hands out its slots in order")
    ras = cr.ComputeRasteriser(ctx)
    ras.addPointCloud(cloud)
    # Every point gets its gradient: no level of detail.
    ras.configuration = cr.ComputeRasteriserConfiguration(enableCLOD=False)
    ras.resize((c["w"], c["h"]))
    images, grad = torch.empty_like(targets), torch.empty_like(colors)
    dimage = torch.empty_like(targets[0])

    def buf(t):
        return cr.DeviceView(ctx, t.data_ptr(), t.shape, np.float32, t)

    return {"ctx": ctx, "ras": ras, "cloud": cloud, "cameras": cams, "images": images,
            "grad": grad, "stream": torch.cuda.ExternalStream(ctx.stream()),
            "scale": 1.0 / targets.numel(), "colors": buf(colors), "grad_buf": buf(grad),
            "dimage": buf(dimage), "views": [(buf(i), buf(t)) for i, t in zip(images, targets)]}


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    return globals()["_run_" + state["kind"]](state)


def _run_frame(s):
    ras = s["ras"]
    ras.update(s["camera"])
    ras.encode()
    if "planes" in s:
        return s["planes"]
    image = s["images"][s["turn"]]
    s["turn"] ^= 1
    ras.outputRGBA8Async(image.numpy())
    ras.waitOutput(1)  # the frame before: its buffer is the next one's
    return {"image": image}


def _run_views(s):
    mv = s["mv"]
    mv.render(s["cameras"])
    images = s["images"][s["turn"]]
    s["turn"] ^= 1
    for f, a in zip(mv.frames, images):
        f.rgba8_async(a.numpy())
    for f in mv.frames:
        f.wait(1)  # the set before, whose buffers are the next one's
    return images


def _run_pick(s):
    k = s["ras"].pickPointIndex(s["at"], s["cloud"], s["camera"])
    return {"index": -1 if k is None else k}


def _run_pack(s):
    s["packer"].pack(into=s["cloud"], **s["raw"])
    return s["pool"]


def _run_chunks(s):
    s["cloud"].clearAllBatches()
    first = s["cloud"].addRawChunksGPU(s["packer"], s["nodes"])
    return dict(s["pool"], first=np.array(first, np.int64))


def _run_train(s):
    ras, cloud = s["ras"], s["cloud"]
    with torch.cuda.stream(s["stream"]):
        s["grad"].zero_()
    for camera, (image, target) in zip(s["cameras"], s["views"]):
        ras.update(camera)
        ras.forwardF32(cloud, s["colors"], image)
        cr.l2_loss(s["ctx"], image, target, s["scale"], s["dimage"], want_loss=False)
        ras.backwardColors(cloud, s["dimage"], s["grad_buf"])
    return {"grad": s["grad"], "images": s["images"]}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    n, kind = case["points"], case["kind"]
    if kind == "pack":  # raw points in, packed points out
        return {"bytes": n * ((16 if case["records"] else 28) + 17), "flops": 0}
    if kind == "chunks":
        return {"bytes": case["chunks"] * n * (28 + 17), "flops": 0}
    if kind == "train":
        # A terrain view holds about a tenth of the field: its points' two
        # words, colour and gradient, and the pixels' image and target.
        seen, px = n * 0.1, case["w"] * case["h"]
        return {"bytes": case["views"] * (seen * (8 + 12 + 12) + px * 24), "flops": 0}
    if kind == "views":
        seen, px = n * 0.2, 900_000
        return {"bytes": case["views"] * (seen * 13 + px * 4 + n / BATCH * 64), "flops": 0}
    # A frame: every batch's record; of the points of a view (about a fifth of
    # a terrain of 100 million, all of the lattice) a level byte, two words
    # and a colour; the image.
    seen = n if case.get("scene") == "lattice" else n * 0.2
    extra = 32 if case.get("effects") else 0
    return {"bytes": n / BATCH * 64 + seen * (13 + extra) + case["w"] * case["h"] * 4, "flops": 0}


# ---------------------------------------------------------------------------
# The training step in 64 bits.  Which pixel a point falls in and whether it
# is seen there are 32-bit decisions of the path (single products and sums,
# no contraction); the sums of colours and gradients are what is computed.
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] != "train":
        return None  # whole numbers and bytes
    mn, mx, words, land = _packed(case, seed)
    colors, targets, cams = _train_inputs(case, seed, land)
    colors, scale = colors.double(), 1.0 / targets.numel()
    nb = mn.shape[0]
    w, h = case["w"], case["h"]
    grad = torch.zeros_like(colors)
    images = torch.zeros(targets.shape, dtype=torch.float64, device="cuda")
    one_less = float(np.float32(1.0) - np.float32(0.01))  # the default depth tolerance
    for v, cam in enumerate(cams):
        view, proj = cam.viewMatrix, cam.projectionMatrix
        t = _product(proj, view)
        px = _pixel_size(mn, mx, view, proj, w, h)
        fine = px >= 500.0  # two words of ten bits from this size on the screen, else one
        if bool((px >= 10000.0).any()):
            fine3 = px >= 10000.0
        else:
            fine3 = torch.zeros_like(fine)
        ix, iy, nz, ok = _project(mn, mx, words, t, fine, fine3, w, h)
        at = torch.nonzero(ok).reshape(-1)
        pix = (h - 1 - iy[at]) * w + ix[at]
        z = nz[at]
        depth = (z * 4294967296.0).to(torch.int64).clamp(0, 4294967295)
        near = torch.zeros(w * h, dtype=torch.int64, device="cuda")
        near.scatter_reduce_(0, pix, depth, "amax")
        closest = near[pix]
        seen = (closest != 0) & (z >= closest.float() / 4294967296.0 * one_less)
        at, pix = at[seen], pix[seen]
        count = torch.zeros(w * h, dtype=torch.float64, device="cuda")
        count.index_add_(0, pix, torch.ones_like(pix, dtype=torch.float64))
        image = torch.zeros((w * h, 3), dtype=torch.float64, device="cuda")
        image.index_add_(0, pix, colors[at])
        image /= count.clamp(min=1.0)[:, None]
        images[v] = image.reshape(h, w, 3)
        d = 2.0 * scale * (image - targets[v].double().reshape(-1, 3))
        grad[at] += d[pix] / count[pix][:, None]
        del ix, iy, nz, ok
    return {"grad": grad, "images": images}


def _product(a, b):
    a, b = (np.asarray(m, np.float32).reshape(4, 4) for m in (a, b))
    out = np.zeros((4, 4), np.float32)
    for c in range(4):
        s = a[0] * b[c, 0] + a[1] * b[c, 1]
        s = s + a[2] * b[c, 2]
        out[c] = s + a[3] * b[c, 3]
    return out.reshape(16)


def _rows(m, x, y, z):
    """A column-major matrix times (x, y, z, 1), in 32 bits, left to right."""
    m = [float(v) for v in m]
    return [((x * m[r] + y * m[4 + r]) + z * m[8 + r]) + m[12 + r] for r in range(4)]


def _pixel_size(mn, mx, view, proj, w, h):
    """A batch's size on the screen: its diagonal at its centre."""
    c = (mn + mx) * 0.5
    r = (mn - mx).square()
    r = ((r[:, 0] + r[:, 1]) + r[:, 2]).sqrt()
    vc = _rows(view, c[:, 0], c[:, 1], c[:, 2])
    pc, pe = _rows(proj, vc[0], vc[1], vc[2]), _rows(proj, vc[0] + r, vc[1], vc[2])
    wc, we = pc[3].abs().clamp(min=1e-6), pe[3].abs().clamp(min=1e-6)
    ex = (w * (pe[0] / we + 1.0)) * 0.5 - (w * (pc[0] / wc + 1.0)) * 0.5
    ey = (h * (pe[1] / we + 1.0)) * 0.5 - (h * (pc[1] / wc + 1.0)) * 0.5
    return (ex * ex + ey * ey).sqrt()


def _project(mn, mx, words, t, fine, fine3, w, h):
    """Pixel column and row (row 0 at the bottom), depth and validity of every point."""
    nb = mn.shape[0]
    low, med, high = (a.reshape(nb, BATCH) for a in words)
    bits = torch.where(fine3, 30, torch.where(fine, 20, 10))
    step = torch.clamp(mx - mn, min=1e-6) / torch.pow(2.0, bits.float())[:, None]
    p = []
    for k in range(3):
        a, b, c = ((q >> (10 * k)) & 1023 for q in (low, med, high))
        q = torch.where(fine3[:, None], (a << 20) | (b << 10) | c,
                        torch.where(fine[:, None], (a << 10) | b, a))
        p.append((q.float() * step[:, k, None] + mn[:, k, None]).reshape(-1))
    cx, cy, cz, cw = _rows(t, *p)
    ok = cw > 0.0
    cw = torch.where(ok, cw, torch.ones_like(cw))
    nx, ny, nz = cx / cw, cy / cw, cz / cw
    ok &= (nx.abs() <= 1.0) & (ny.abs() <= 1.0) & (nz >= 0.0) & (nz <= 1.0)
    nx, ny = torch.where(ok, nx, torch.zeros_like(nx)), torch.where(ok, ny, torch.zeros_like(ny))
    ix, iy = ((nx * 0.5 + 0.5) * w).to(torch.int64), ((ny * 0.5 + 0.5) * h).to(torch.int64)
    ok &= (ix < w) & (iy < h)
    return ix, iy, nz, ok
