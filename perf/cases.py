"""Workloads of the renderer, for timing one pass through its public entry points.

A case is a dict of plain values.  ``path`` names the entry point:

* ``view``     one ``Renderer.render`` call (bricks resident, a new image per call);
* ``sampler``  yt's call surface: a ``VolumeRenderSampler`` built, called once per brick
               with host arrays, and its ``aimage`` read;
* ``batch``    many views of resident volumes, replayed as a CUDA graph;
* ``octree``   one ``render_octree`` launch over a resident octree;
* ``offaxis``  one ``CellSplat.project`` call over resident cells.

The data are the generators the tests and the benchmark use in kind: Gaussian blobs
times lognormal noise, refined by factor 2 in 16^3 patches, and lognormal random
fields.  ``exact`` renders the same inputs in float64 with torch alone, by marching
each ray from cell face to cell face.
"""
import math

import numpy as np
import torch

BLOCK = 8  # refinement unit: a block of BLOCK^3 cells becomes a patch of (2 BLOCK)^3
BALL = 0.45  # radius of the masked cases' data source
SAMPLERS = ("vr", "proj", "iproj", "mip", "light")


# ---- the cases ---------------------------------------------------------------------------
def _case(path, **kw):
    """A case with every key its path reads (kw overrides the defaults)."""
    base = {"path": path, "nx": 512, "ny": 512, "theta": 57.0, "phi": 25.0}
    if path in ("view", "sampler"):
        base.update(data="amr", root=64, levels=3, sampler="vr", lens="perspective", samples=1, layers=8,
                    range64=False, grey=False, masked=False)
    elif path == "batch":
        base.update(root=64, levels=3, views=16, layers=8)
    else:
        base.update(base_level=5, max_level=8, sampler="vr", samples=1, layers=8)
    base.update(kw)
    return base


def listed():
    named = [
        # the smallest call: one uniform brick seen through a plane-parallel lens, as in a
        # first look at a dataset (four layers, a preview-sized image)
        ("uniform-vr-256", _case("view", data="uniform", root=64, nx=256, ny=256, lens="plane-parallel", layers=4,
                                 theta=0.0, phi=0.0)),
        # the benchmark frame: a 128^3 root with three refinement levels, perspective
        ("amr-vr-1024", _case("view", root=128, nx=1024, ny=1024)),
        # a volume kept with its float32 rounding errors (what the render server keeps), the
        # transfer function cutting through the data, an odd image
        ("amr-vr-range64", _case("view", root=64, levels=4, nx=701, ny=1003, range64=True, theta=80.0, phi=130.0)),
        # yt's default of ten samples per cell, with a data source that masks cells out
        ("amr-vr-10-samples", _case("view", root=64, nx=640, ny=480, lens="plane-parallel", samples=10, masked=True,
                                    theta=35.0, phi=200.0)),
        # the projection study: a 512^3 random field at 2048^2
        ("projection-2048", _case("view", data="uniform", root=512, nx=2048, ny=2048, sampler="proj",
                                  lens="plane-parallel", theta=30.0)),
        # a maximum projection of an odd grid at an odd size
        ("mip-odd", _case("view", data="uniform", root=255, nx=1023, ny=779, sampler="mip", lens="plane-parallel")),
        # off-axis interpolated projection of AMR data
        ("amr-iproj-1024", _case("view", root=128, nx=1024, ny=768, sampler="iproj", theta=110.0, phi=300.0)),
        # lit volume rendering, grey opacity off, general transfer-function path
        ("amr-light", _case("view", root=64, nx=512, ny=512, sampler="light", theta=45.0, phi=75.0)),
        # sixteen views of mixed size and sampler in one batch (an animation, a served group)
        ("batch-16", _case("batch", root=64, levels=4, views=16, nx=1024)),
        # an octree dataset: rays cast through its cells
        ("octree-vr-1024", _case("octree", base_level=5, max_level=9, nx=1024, ny=1024)),
        # the same kind of dataset projected by splatting its cells
        ("offaxis-1024", _case("offaxis", base_level=5, max_level=9, nx=1024, ny=1024)),
        # the drop-in sampler under yt's Scene.render: host bricks in, host image out
        ("sampler-1024", _case("sampler", root=128, nx=1024, ny=1024, theta=20.0, phi=10.0)),
    ]
    return [dict(c, name=n) for n, c in named]


def _spread(rng, lo, hi):
    """An integer from lo to hi, uniform in its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    path = rng.choice(["view"] * 6 + ["batch", "octree", "offaxis", "sampler"])
    kw = {"nx": _spread(rng, 96, 1024), "ny": _spread(rng, 96, 1024),
          "theta": round(rng.uniform(3.0, 177.0), 3), "phi": round(rng.uniform(1.0, 359.0), 3)}
    if path in ("view", "sampler"):
        kw["sampler"] = rng.choice(SAMPLERS) if path == "view" else "vr"
        kw["data"] = "uniform" if kw["sampler"] in ("proj", "mip") else rng.choice(["uniform", "amr", "amr"])
        kw["root"] = (_spread(rng, 24, 400 if kw["sampler"] in ("proj", "mip") else 160) if kw["data"] == "uniform"
                      else BLOCK * rng.randint(6, 14))
        kw["levels"] = rng.randint(1, 3)
        kw["lens"] = rng.choice(["plane-parallel", "perspective"])
        kw["layers"] = rng.randint(2, 8)
        if kw["sampler"] not in ("proj", "mip"):
            kw["samples"] = rng.choice([1, 1, 1, 2, 10 if kw["data"] == "amr" else 4])
        if kw["sampler"] == "vr":
            kw["grey"] = rng.random() < 0.3
            kw["masked"] = rng.random() < 0.25
            kw["range64"] = path == "view" and not kw["masked"] and rng.random() < 0.3
    elif path == "batch":
        kw.update(root=BLOCK * rng.randint(6, 10), levels=rng.randint(1, 3), views=rng.randint(2, 24),
                  nx=_spread(rng, 128, 800))
    else:
        kw.update(base_level=rng.randint(3, 5), max_level=rng.randint(6, 8), layers=rng.randint(2, 8))
        if path == "octree":
            kw["sampler"] = rng.choice(["vr", "vr", "iproj", "proj", "mip"])
        else:
            kw["nx"], kw["ny"] = min(kw["nx"], kw["ny"]), max(kw["nx"], kw["ny"])
    return _case(path, **kw)


# ---- the data ----------------------------------------------------------------------------
def _blobs(rng):
    return rng.uniform(0.2, 0.8, (8, 3)), rng.uniform(0.05, 0.12, 8), rng.lognormal(0.0, 1.0, 8)


def _density(blobs, axes):
    """1 + a sum of Gaussian blobs on the tensor grid of three coordinate axes."""
    rho = np.ones([a.size for a in axes])
    for c, s, amp in zip(*blobs):
        gx, gy, gz = (np.exp(-((a - x) ** 2) / (2 * s * s)) for a, x in zip(axes, c))
        rho += amp * gx[:, None, None] * gy[None, :, None] * gz[None, None, :]
    return rho


def _amr(root, levels, seed):
    """(level, first cell in units of that level's cells, data) of a root grid of root^3
    cells on [0, 1]^3 and its patches: at each level the blocks whose mean log10 density is
    above the 90th percentile of all blocks are refined."""
    rng = np.random.default_rng(seed)
    blobs = _blobs(rng)

    def grid(level, lo, n):
        dx = 1.0 / (root << level)
        axes = [(lo[i] + np.arange(n) + 0.5) * dx for i in range(3)]
        return level, lo, _density(blobs, axes) * np.exp(0.1 * rng.standard_normal((n, n, n)))

    last = [grid(0, np.zeros(3, np.int64), root)]
    grids = list(last)
    for level in range(1, levels + 1):
        means = []
        for _, _, d in last:
            n = d.shape[0] // BLOCK
            means.append(np.log10(d).reshape(n, BLOCK, n, BLOCK, n, BLOCK).mean(axis=(1, 3, 5)))
        cut = np.percentile(np.concatenate([m.ravel() for m in means]), 90.0)
        last = [grid(level, 2 * (lo + BLOCK * np.array(ijk)), 2 * BLOCK)
                for (_, lo, _), m in zip(last, means) for ijk in np.argwhere(m > cut)]
        grids += last
    return grids


def _random_field(n, seed):
    """A lognormal random field of (n, n + 1, n - 2) cells in float32 values: octaves of
    noise, as one root level of (level, lo, data)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    shape = (n, n + 1, n - 2)
    f = 0.3 * torch.randn(shape, generator=gen, device="cuda")
    m, amp = 4, 0.8
    while m < n:
        noise = torch.randn((1, 1, m, m, m), generator=gen, device="cuda")
        f += amp * torch.nn.functional.interpolate(noise, size=shape, mode="trilinear", align_corners=False)[0, 0]
        m, amp = 2 * m, 0.7 * amp
    return torch.exp(f)


def _mask(le, dx, dims):
    """The cells' mask of a brick for a data source that is a ball: cells whose centre lies
    within BALL of the domain's centre."""
    ax = [(le[i] + (np.arange(dims[i]) + 0.5) * dx[i] - 0.5) ** 2 for i in range(3)]
    return (ax[0][:, None, None] + ax[1][None, :, None] + ax[2][None, None, :] < BALL ** 2).astype(np.uint8)


def _bounds(values, case):
    """The transfer function's bounds: the data's extremes widened a little, or, where range
    decisions are made in float64, bounds that cut through the data."""
    lo, hi = float(values.min()), float(values.max())
    d = 0.03 * (hi - lo)
    return (lo + d, hi - d) if case.get("range64") else (lo - d, hi + d)


def _layers(bounds, n):
    """(location, width, rgba) of n Gaussian layers, alphas from 0.001 to 1."""
    b0, b1 = bounds
    d = b1 - b0
    out = []
    for v, a in zip(np.linspace(b0 + d / (10 * n), b1 - d / (10 * n), n), np.logspace(-3, 0, n)):
        s = (v - b0) / d
        out.append((float(v), 0.01, (min(1.5 * s + 0.1, 1.0), 1.0 - abs(2 * s - 1.0), 1.0 - 0.8 * s, float(a))))
    return out


def _octree(case, seed):
    """(level, integer position, corner values) of each leaf cell, level by level: a cell is
    refined where the field at its centre is above the 85th percentile of its level."""
    rng = np.random.default_rng(seed)
    blobs = _blobs(rng)

    def at(x):
        v = np.ones(x.shape[:-1])
        for c, s, amp in zip(*blobs):
            v += amp * np.exp(-((x - c) ** 2).sum(-1) / (2 * s * s))
        return v

    n = 1 << case["base_level"]
    corners = np.stack(np.meshgrid(*[np.arange(2)] * 3, indexing="ij"), -1).reshape(8, 3)
    idx = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)
    level, out = case["base_level"], []
    while True:
        dx = 1.0 / (1 << level)
        val = at((idx + 0.5) * dx)
        refine = val > np.percentile(val, 85.0) if level < case["max_level"] else np.zeros(val.size, bool)
        keep = idx[~refine]
        out.append((level, keep, np.log10(at((keep[:, None] + corners[None]) * dx))))
        if level == case["max_level"]:
            return out
        idx = (2 * idx[refine][:, None] + corners[None]).reshape(-1, 3)
        level += 1


# ---- cameras -----------------------------------------------------------------------------
def _geometry(case, theta=None, phi=None):
    """(position, width, north) of a camera that looks at the domain's centre."""
    t, p = math.radians(case["theta"] if theta is None else theta), math.radians(case["phi"] if phi is None else phi)
    normal = np.array([math.sin(t) * math.cos(p), math.sin(t) * math.sin(p), math.cos(t)])
    width = 1.1 if case.get("lens") == "plane-parallel" else 1.5
    return np.array([0.5, 0.5, 0.5]) - 1.5 * normal, width, (0.31, 0.9, 0.17)


def _camera(case, lens, nx, ny, theta=None, phi=None):
    from yt_gb300.camera import Camera

    pos, width, north = _geometry(case, theta, phi)
    return Camera(pos, (0.5, 0.5, 0.5), width, (nx, ny), north_vector=north, lens_type=lens)


def _views(case):
    """(sampler, size, theta, phi) of a batch's views: points of a spiral on the sphere, image
    sizes from an eighth of nx up to nx, every third an interpolated projection."""
    out = []
    for k in range(case["views"]):
        size = max(32, int(case["nx"] / (1, 2, 4, 3, 8)[k % 5]))
        out.append(("iproj" if k % 3 == 2 else "vr", size,
                    math.degrees(math.acos(1 - 2 * (k + 0.5) / case["views"])), (case["phi"] + 137.508 * k) % 360.0))
    return out


# ---- what a program has in hand before the call --------------------------------------------
def _tf(bounds, case):
    from yt_gb300.transfer_functions import ColorTransferFunction

    tf = ColorTransferFunction(bounds, grey_opacity=bool(case.get("grey")))
    for loc, w, rgba in _layers(bounds, case["layers"]):
        tf.add_gaussian(loc, w, list(rgba))
    return tf


def _uniform(case, seed):
    """The one grid of a uniform case: cell values (root^3 blobs for the interpolating
    samplers, a random field for the cell samplers)."""
    if case["sampler"] in ("proj", "mip"):
        return _random_field(case["root"], seed).double().cpu().numpy()
    rng = np.random.default_rng(seed)
    blobs, n = _blobs(rng), case["root"]
    ax = (np.arange(n) + 0.5) / n
    return _density(blobs, [ax, ax, ax]) * np.exp(0.1 * rng.standard_normal((n, n, n)))


def _volume(case, seed):
    """(kd-tree or None, cell-centred field or None, transfer function)."""
    from yt_gb300 import testing
    from yt_gb300.amr_kdtree import AMRKDTree

    if case.get("sampler") in ("proj", "mip"):
        return None, _uniform(case, seed), None
    if case.get("data") == "uniform":
        grids = [(0, np.zeros(3, np.int64), _uniform(case, seed))]
        root = case["root"]
    else:
        root = case["root"]
        grids = _amr(root, case["levels"], seed)
    objs = []
    for k, (lv, lo, d) in enumerate(grids):
        n = root << lv
        objs.append(testing.Grid(k, lv, lo / n, (lo + d.shape[0]) / n, np.array(d.shape, np.int64), d))
    log = case.get("sampler") != "iproj"
    first = np.log10(grids[0][2]) if log else grids[0][2]
    return AMRKDTree(objs, log_field=log), None, _tf(_bounds(first, case), case)


def _masked(kd):
    out = []
    for data, _, le, re, dims in kd.bricks():
        out.append((data, _mask(le, (re - le) / dims, dims), le, re, dims))
    return out


def _prepare_view(case, seed):
    from yt_gb300 import _lib
    from yt_gb300.render import Renderer

    kind = {"vr": _lib.VOLUME_RENDER, "proj": _lib.PROJECTION, "iproj": _lib.INTERPOLATED_PROJECTION,
            "mip": _lib.MIP, "light": _lib.LIGHT_SOURCE}[case["sampler"]]
    kd, field, tf = _volume(case, seed)
    if field is not None:
        bricks = [([field], None, np.zeros(3), np.ones(3), np.array(field.shape, np.int64))]
    elif case["masked"]:
        bricks = _masked(kd)
    else:
        bricks = kd.device_brickset(with_lo=case["range64"])
    r = Renderer(bricks, tf, kdtree=kd)
    light = ((1.0, 0.4, -0.3), (0.9, 0.8, 0.7, 1.0)) if case["sampler"] == "light" else None
    return {"renderer": r, "camera": _camera(case, case["lens"], case["nx"], case["ny"]), "kind": kind, "light": light,
            "samples": case["samples"]}


def _prepare_sampler(case, seed):
    kd, _, tf = _volume(case, seed)
    from yt_gb300.partitioned_grid import PartitionedGrid

    cam = _camera(case, case["lens"], case["nx"], case["ny"])
    p = cam.sampler_params()
    if case["masked"]:
        bricks = _masked(kd)
        order = kd.viewpoint_order(cam.viewpoint)
        grids = [PartitionedGrid(k, *bricks[k]) for k in order]
    else:
        grids = list(kd.traverse(cam.viewpoint))
    return {"params": p, "tf": tf, "bricks": grids, "samples": case["samples"]}


def _prepare_batch(case, seed):
    from yt_gb300 import _lib
    from yt_gb300.batch import Batch, Job
    from yt_gb300.render import Renderer

    kd, _, tf = _volume(case, seed)
    r = Renderer(kd.device_brickset(), tf, kdtree=kd)
    kinds = {"vr": _lib.VOLUME_RENDER, "iproj": _lib.INTERPOLATED_PROJECTION}
    batch = Batch([Job(r, _camera(case, "perspective", n, n, t, p), kinds[s]) for s, n, t, p in _views(case)])
    return {"batch": batch, "graph": batch.capture()}


def _prepare_octree(case, seed):
    from yt_gb300 import _lib
    from yt_gb300.octree import Octree, OctreeVolume
    from yt_gb300.transfer_functions import pack

    ipos, lvl, rows = [], [], []
    depth = case["max_level"]
    for lv, ix, v in _octree(case, seed):
        dx = 1.0 / (1 << lv)
        ipos.append(np.floor((ix + 0.5) * dx * (1 << depth)).astype(np.int32))
        lvl.append(np.full(len(ix), lv, np.int32))
        rows.append(np.concatenate([v, ix * dx, ix * dx + dx], axis=1))
    cells = np.concatenate(rows)
    tree = Octree(np.zeros(3), np.ones(3), depth)
    tree.add_nodes(np.concatenate(ipos), np.concatenate(lvl), np.arange(len(cells), dtype=np.int32))
    kind = {"vr": _lib.VOLUME_RENDER, "proj": _lib.PROJECTION, "iproj": _lib.INTERPOLATED_PROJECTION,
            "mip": _lib.MIP}[case["sampler"]]
    view = _camera(case, "perspective", case["nx"], case["ny"]).device_view()
    return {"volume": OctreeVolume(tree, cells), "view": view, "kind": kind, "size": (case["nx"], case["ny"], 4),
            "tf": pack(_tf(_bounds(cells[:, :8], case), case)), "samples": case["samples"]}


def _splat(case, seed):
    """(cell centres about the image's centre, widths, quantity, weight, rotation)."""
    x, dx, q = [], [], []
    for lv, ix, v in _octree(case, seed):
        h = 1.0 / (1 << lv)
        x.append((ix + 0.5) * h - 0.5)
        dx.append(np.full(len(ix), h))
        q.append(v.mean(axis=1))
    rng = np.random.default_rng(seed + 1)
    x, dx, q = np.concatenate(x), np.concatenate(dx), np.concatenate(q)
    t, p = math.radians(case["theta"]), math.radians(case["phi"])
    rx = np.array([[1, 0, 0], [0, math.cos(t), -math.sin(t)], [0, math.sin(t), math.cos(t)]])
    rz = np.array([[math.cos(p), -math.sin(p), 0], [math.sin(p), math.cos(p), 0], [0, 0, 1]])
    return x / 1.5, dx / 1.5, q, rng.uniform(0.5, 1.5, q.size), rx @ rz  # an image 1.5 domains wide


def _prepare_offaxis(case, seed):
    from yt_gb300.offaxis import CellSplat

    x, dx, q, w, rot = _splat(case, seed)
    s = CellSplat(x, dx, q, w)
    s.stamp(rot, case["nx"], case["ny"])  # kept by the cells for this view
    return {"splat": s, "rotation": rot, "nx": case["nx"], "ny": case["ny"]}


def prepare(case, seed):
    state = {"view": _prepare_view, "sampler": _prepare_sampler, "batch": _prepare_batch, "octree": _prepare_octree,
             "offaxis": _prepare_offaxis}[case["path"]](case, seed)
    state["path"] = case["path"]
    return state


def run(state):
    if state["path"] == "view":
        return state["renderer"].render(state["camera"], kind=state["kind"], n_samples=state["samples"],
                                        light=state["light"])
    if state["path"] == "batch":
        state["graph"].replay()
        return state["batch"].images
    if state["path"] == "octree":
        from yt_gb300.octree import render_octree

        image = torch.zeros(state["size"], dtype=torch.float64, device="cuda")
        render_octree(state["volume"], state["view"], state["kind"], image, tf=state["tf"],
                      n_samples=state["samples"])
        return image
    if state["path"] == "offaxis":
        return state["splat"].project(state["rotation"], state["nx"], state["ny"])
    from yt_gb300.image_samplers import VolumeRenderSampler

    p = state["params"]
    s = VolumeRenderSampler(np.atleast_3d(p["vp_pos"]), np.atleast_3d(p["vp_dir"]), p["center"], p["bounds"],
                            np.zeros(p["image"].shape), p["x_vec"], p["y_vec"], p["width"], "KDTree", state["tf"],
                            state["samples"], lens_type=p["lens_type"], camera_data=p["camera_data"])
    for pg in state["bricks"]:
        s(pg)
    return s.aimage


# ---- what a pass cannot do without ---------------------------------------------------------
def _cells_along(case):
    """About how many cells one ray of the case meets."""
    if case["path"] == "octree":
        return 1.2 * (1 << case["base_level"]) * (1 + 0.25 * (case["max_level"] - case["base_level"]))
    if case.get("data") == "uniform":
        return 1.2 * case["root"]
    return 1.2 * case["root"] * (1 + 0.3 * case["levels"])


def work(case):
    rays = case["nx"] * case["ny"]
    if case["path"] == "batch":
        rays = sum(n * n for _, n, _, _ in _views(case))
    if case["path"] in ("octree", "offaxis"):
        cells = (1 << (3 * case["base_level"])) * (1 + 1.2 * (case["max_level"] - case["base_level"]))
    elif case.get("data") == "uniform":
        cells = case["root"] ** 3
    else:
        cells = case["root"] ** 3 * (1 + 0.8 * case["levels"])
    if case["path"] == "offaxis":  # six float64 values a cell, two images; a few operations a pixel touched
        return {"bytes": 48 * cells + 16 * rays, "flops": 30 * cells * max(1.0, rays * 3.0 / 4 ** case["max_level"])}
    per_cell = {"proj": 3, "mip": 2}.get(case.get("sampler"))
    if per_cell is None:
        per_cell = 60 * case.get("samples", 1)
    host = 8 if case["path"] == "sampler" else 4
    hit = 0.5
    return {"bytes": host * cells + 32 * rays, "flops": hit * rays * _cells_along(case) * (per_cell + 10)}


# ---- the same images in float64, with torch alone ------------------------------------------
def _rays(case, lens, nx, ny, theta=None, phi=None):
    """(origin, direction) of every pixel, (nx * ny, 3), as yt's lenses define them."""
    pos, width, north = _geometry(case, theta, phi)
    dev = "cuda"
    normal = np.array([0.5, 0.5, 0.5]) - pos
    normal /= math.sqrt(normal @ normal)
    north = np.array(north) - (np.array(north) @ normal) * normal
    east = np.cross(north, normal)
    north, east = north / math.sqrt(north @ north), east / math.sqrt(east @ east)
    e, n, w = (torch.tensor(v, dtype=torch.float64, device=dev) for v in (east, north, normal))
    i = torch.arange(nx, dtype=torch.float64, device=dev)[:, None, None]
    j = torch.arange(ny, dtype=torch.float64, device=dev)[None, :, None]
    if lens == "plane-parallel":
        px, py = width * i / (nx - 1) - width / 2, width * j / (ny - 1) - width / 2
        o = e * px + n * py + torch.tensor(np.full(3, 0.5) - 0.5 * width * normal, device=dev)
        d = (w * width).expand_as(o)
    else:
        px, py = i / (nx - 1) - 0.5, j / (ny - 1) - 0.5
        scale = (math.sqrt(((pos - 0.5) ** 2).sum()) + 0.5 * math.sqrt(3.0)) / width
        d = (e * (width * px) + n * (width * ny / nx * py) + w * width) * scale
        o = torch.tensor(pos, device=dev).expand_as(d)
    return o.reshape(-1, 3).contiguous(), d.reshape(-1, 3).contiguous()


def _vertices(c, log):
    """Vertex values of a block of cells: averages of the eight cells around, extrapolated
    linearly at the block's faces."""
    for ax in range(3):
        c = np.moveaxis(c, ax, 0)
        mid = 0.5 * (c[1:] + c[:-1])
        c = np.concatenate([(1.5 * c[0] - 0.5 * c[1])[None], mid, (1.5 * c[-1] - 0.5 * c[-2])[None]])
        c = np.moveaxis(c, 0, ax)
    if log:
        with np.errstate(invalid="ignore", divide="ignore"):
            c = np.log10(np.where(c > 0, c, np.nan))
    return c


def _scene(case, seed):
    """Grids as device tables: a lookup of the finest grid over a uniform table, and per grid
    its left edge, cell width, dims, and where its values begin."""
    dev = "cuda"
    if case["path"] == "octree":
        depth = case["max_level"]
        n = 1 << depth
        table = torch.empty((n, n, n), dtype=torch.int32, device=dev)
        le, dx, vals, first = [], [], [], 0
        for lv, ix, v in _octree(case, seed):
            s = 1 << (depth - lv)
            t = torch.from_numpy(ix * s).to(dev)
            ids = torch.arange(first, first + len(ix), dtype=torch.int32, device=dev)
            for q in range(s ** 3):
                table[t[:, 0] + q // (s * s), t[:, 1] + q // s % s, t[:, 2] + q % s] = ids
            first += len(ix)
            le.append(ix / (1 << lv))
            dx.append(np.full((len(ix), 3), 1.0 / (1 << lv)))
            vals.append(v)
        le, dx, vals = np.concatenate(le), np.concatenate(dx), np.concatenate(vals)
        bounds = _bounds(vals, case)
        dims = np.ones_like(le, dtype=np.int64)
        off = 8 * np.arange(len(le))
        return _on_device(table, le, dx, dims, off, torch.from_numpy(vals).to(dev).reshape(-1), None, True, bounds)
    if case.get("sampler") in ("proj", "mip"):
        f = _random_field(case["root"], seed).double()
        shape = np.array([f.shape])
        return _on_device(torch.zeros((1, 1, 1), dtype=torch.int32, device=dev), np.zeros((1, 3)), 1.0 / shape, shape,
                          np.zeros(1, np.int64), f.reshape(-1), None, False, None)
    root = case["root"]
    if case.get("data") == "uniform":
        grids = [(0, np.zeros(3, np.int64), _uniform(case, seed))]
        table = torch.zeros((1, 1, 1), dtype=torch.int32, device=dev)
    else:
        grids = _amr(root, case["levels"], seed)
        top = max(lv for lv, _, _ in grids)
        n = (root // BLOCK) << top
        table = np.zeros((n, n, n), np.int32)
        for k, (lv, lo, d) in enumerate(grids):
            a = (lo // BLOCK) << (top - lv)
            m = (d.shape[0] // BLOCK) << (top - lv)
            table[a[0]:a[0] + m, a[1]:a[1] + m, a[2]:a[2] + m] = k
        table = torch.from_numpy(table).to(dev)
    log = case.get("sampler") != "iproj"
    verts = [_vertices(d, log).ravel() for _, _, d in grids]
    le = np.array([lo / (root << lv) for lv, lo, _ in grids])
    dx = np.array([[1.0 / (root << lv)] * 3 for lv, _, _ in grids])
    dims = np.array([d.shape for _, _, d in grids], dtype=np.int64)
    off = np.concatenate([[0], np.cumsum([v.size for v in verts])[:-1]])
    first = np.log10(grids[0][2]) if log else grids[0][2]
    ball = BALL if case.get("masked") else None
    return _on_device(table, le, dx, dims, off, torch.from_numpy(np.concatenate(verts)).to(dev), ball, True,
                      _bounds(first, case))


def _on_device(table, le, dx, dims, off, vals, ball, vertex, bounds):
    t = {k: torch.from_numpy(np.ascontiguousarray(v)).to("cuda") for k, v in
         (("le", le), ("dx", dx), ("dims", dims), ("off", off))}
    return dict(t, table=table, vals=vals, ball=ball, vertex=vertex, bounds=bounds)


def _emission(v, bounds, case):
    """(rgb emission times alpha, alpha) of sample values from tables of 256 bins."""
    b0, b1 = bounds
    x = np.linspace(b0, b1, 256)
    y = np.zeros((4, 256))
    for loc, w, rgba in _layers(bounds, case["layers"]):
        for c in range(4):
            y[c] = np.maximum(y[c], rgba[c] * np.exp(-((x - loc) ** 2) / w))
    dy = (y[:, 1:] - y[:, :-1]) / (x[1:] - x[:-1])
    y, dy, x = (torch.from_numpy(a).to(v.device) for a in (y, dy, x))
    inside = (v > b0) & (v < b1) & (v != 0)
    s = torch.where(inside, v, torch.full_like(v, b0))
    bin_ = ((s - b0) * (255 / (b1 - b0))).floor().clamp(0, 254).long()
    t = y[:, bin_] + (s - x[bin_]) * dy[:, bin_]
    t = torch.where(inside, t, torch.zeros_like(t))
    return t[:3] * t[3], t[3]


def _march(o, d, sc, case, sampler, ns, light=None):
    """The image of rays o + t d, t in [0, 1], through a scene, cell by cell, front to back."""
    image = torch.zeros((o.shape[0], 4), dtype=torch.float64, device=o.device)
    ta, tb = (0.0 - o) / d, (1.0 - o) / d
    t0 = torch.minimum(ta, tb).amax(1).clamp(min=0.0)
    t1 = torch.maximum(ta, tb).amin(1).clamp(max=1.0)
    live = torch.nonzero(t1 > t0)[:, 0]
    x, p, v, t, end = image[live], o[live], d[live], t0[live], t1[live]
    tiny = 1e-12
    size = torch.tensor(sc["table"].shape, device=o.device)
    step = 0
    while live.numel():
        at = p + v * (t + tiny)[:, None]
        b = (at * size).floor().long()
        b = torch.minimum(b.clamp(min=0), size - 1)
        g = sc["table"][b[:, 0], b[:, 1], b[:, 2]].long()
        le, dx, dims = sc["le"][g], sc["dx"][g], sc["dims"][g]
        c = torch.minimum(((at - le) / dx).floor().long().clamp(min=0), dims - 1)
        face = le + (c + (v > 0)) * dx
        te = torch.where(v != 0, (face - p) / v, torch.full_like(v, math.inf)).amin(1)
        te = torch.minimum(torch.maximum(te, t), end)
        dt = te - t
        if sc["vertex"]:
            m = dims + 1
            i0 = sc["off"][g] + (c[:, 0] * m[:, 1] + c[:, 1]) * m[:, 2] + c[:, 2]
            sx, sy = m[:, 1] * m[:, 2], m[:, 2]
            q = [sc["vals"][i0 + a * sx + b2 * sy + e] for a in (0, 1) for b2 in (0, 1) for e in (0, 1)]
        else:
            val = sc["vals"][sc["off"][g] + (c[:, 0] * dims[:, 1] + c[:, 1]) * dims[:, 2] + c[:, 2]]
        for s in range(ns):
            if sc["vertex"]:
                f = (p + v * (t + (s + 0.5) * dt / ns)[:, None] - (le + c * dx)) / dx
                fx, fy, fz = f[:, 0], f[:, 1], f[:, 2]
                z = [q[2 * k] + fz * (q[2 * k + 1] - q[2 * k]) for k in range(4)]
                y0, y1 = z[0] + fy * (z[1] - z[0]), z[2] + fy * (z[3] - z[2])
                val = q[0] if sampler in ("proj", "mip") else y0 + fx * (y1 - y0)  # (an octree cell's first value)
            h = dt / ns
            if sampler in ("proj", "iproj"):
                x[:, 0] += val * h
            elif sampler == "mip":
                x[:, 0] = torch.maximum(x[:, 0], val)
            else:
                e, al = _emission(val, sc["bounds"], case)
                if sampler == "light":
                    gx = y1 - y0
                    gy = (z[1] - z[0]) + fx * ((z[3] - z[2]) - (z[1] - z[0]))
                    dz = [q[2 * k + 1] - q[2 * k] for k in range(4)]
                    d0, d1 = dz[0] + fy * (dz[1] - dz[0]), dz[2] + fy * (dz[3] - dz[2])
                    gz = d0 + fx * (d1 - d0)
                    n = torch.sqrt(gx * gx + gy * gy + gz * gz)
                    ld = np.array(light[0]) / math.sqrt(sum(u * u for u in light[0]))
                    dot = -(ld[0] * gx + ld[1] * gy + ld[2] * gz) / n
                    for ch in range(3):
                        keep = (1 - h * e[ch]).clamp(min=0)
                        x[:, ch] = (1 - keep) * e[ch] * (1 + dot * light[1][ch]) + keep * x[:, ch]
                else:
                    new = x.clone()
                    for ch in range(4 if case.get("grey") else 3):
                        em = h * (e[ch] if ch < 3 else al)
                        keep = (1 - (h * al if case.get("grey") else em)).clamp(min=0)
                        new[:, ch] = em + keep * x[:, ch]
                    if sc["ball"] is not None:
                        ctr = le + (c + 0.5) * dx - 0.5
                        new = torch.where(((ctr * ctr).sum(1) < sc["ball"] ** 2)[:, None], new, x)
                    x = new
        t = torch.maximum(te, t + tiny)
        step += 1
        if step % 8 == 0:
            image[live] = x
            on = torch.nonzero(t < end - tiny)[:, 0]
            live, x, p, v, t, end = live[on], x[on], p[on], v[on], t[on], end[on]
        else:
            end = torch.where(t < end - tiny, end, t)  # a finished ray takes steps of no length
    return image


def _exact_splat(case, seed):
    """Every cell's projected cube cut into subcells of the stamp and spread bilinearly."""
    x, dx, q, w, rot = _splat(case, seed)
    nx, ny, dev = case["nx"], case["ny"], "cuda"
    r3 = math.sqrt(3.0)
    nsx, nsy = (max(4, math.ceil(2 * dx.max() * r3 * n)) for n in (nx, ny))
    levels = math.ceil(math.log2(max(nsx, nsy)))
    depth = np.clip(np.ceil(np.log2(4 * r3 * dx * max(nx, ny))).astype(int), 1, levels - 1)
    scr = x @ rot[:2].T + 0.5
    out = [torch.zeros(nx * ny, dtype=torch.float64, device=dev) for _ in range(2)]
    for k in np.unique(depth):
        m = (min(nsx, 1 << k), min(nsy, 1 << k))
        u, v = ((torch.arange(n, dtype=torch.float64, device=dev) + 0.5) / n - 0.5 for n in m)
        lo = torch.full(m, -math.inf, dtype=torch.float64, device=dev)
        hi = -lo
        for i in range(3):  # the cube's three slabs along the line of sight
            s = rot[0, i] * u[:, None] + rot[1, i] * v[None, :]
            a, b = (-0.5 / r3 - s) / rot[2, i], (0.5 / r3 - s) / rot[2, i]
            lo, hi = torch.maximum(lo, torch.minimum(a, b)), torch.minimum(hi, torch.maximum(a, b))
        stamp = (hi - lo).clamp(min=0)
        stamp /= stamp.sum()
        sel = np.nonzero(depth == k)[0]
        for part in np.array_split(sel, max(1, sel.size * m[0] * m[1] // 8_000_000)):
            axes = []
            for ax, n in ((0, nx), (1, ny)):
                i = torch.arange(m[ax] + 1, dtype=torch.float64, device=dev)
                size = torch.from_numpy(dx[part] * r3 / m[ax]).to(dev)[:, None]
                b = ((i - m[ax] / 2.0) * size + torch.from_numpy(scr[part, ax]).to(dev)[:, None]) * n
                e = b.trunc()
                f = ((e[:, 1:] - b[:, :-1]) / (b[:, 1:] - b[:, :-1])).clamp(0, 1)
                axes.append([(e[:, :-1].long(), f), (e[:, 1:].long(), 1 - f)])
            scale = torch.from_numpy(dx[part] ** 3 * nx * ny).to(dev)
            for pi, fx in axes[0]:
                for pj, fy in axes[1]:
                    ok = ((pi >= 0) & (pi < nx))[:, :, None] & ((pj >= 0) & (pj < ny))[:, None, :]
                    idx = (pi[:, :, None] * nx + pj[:, None, :])
                    ok &= idx < nx * ny
                    mass = fx[:, :, None] * fy[:, None, :] * stamp * scale[:, None, None]
                    mass = torch.where(ok, mass, torch.zeros_like(mass))
                    idx = torch.where(ok, idx, torch.zeros_like(idx)).reshape(-1)
                    for buf, val in zip(out, (q, w)):
                        m3 = mass * torch.from_numpy(val[part]).to(dev)[:, None, None]
                        buf.index_add_(0, idx, m3.reshape(-1))
    return tuple(out)


def exact(case, seed):
    if case["path"] == "offaxis":
        return _exact_splat(case, seed)
    sc = _scene(case, seed)
    if case["path"] == "batch":
        out = []
        for s, n, t, p in _views(case):
            o, d = _rays(case, "perspective", n, n, t, p)
            out.append(_march(o, d, sc, case, s, 1).reshape(n, n, 4))
        return out
    lens = case.get("lens", "perspective")
    o, d = _rays(case, lens, case["nx"], case["ny"])
    light = ((1.0, 0.4, -0.3), (0.9, 0.8, 0.7, 1.0))
    parts = [_march(a, b, sc, case, case["sampler"], case["samples"], light)
             for a, b in zip(o.split(1 << 21), d.split(1 << 21))]
    return torch.cat(parts).reshape(case["nx"], case["ny"], 4)
