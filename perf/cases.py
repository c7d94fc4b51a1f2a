"""Workloads for timing the framework through its Python entry points.

`listed()` names the workloads, `draw(rng)` makes more of the same ranges, `prepare(case, seed)` makes what a program
has in hand before the call (meshes, rays, the trees and buffers it keeps), `run(state)` is one pass, `work(case)` the
bytes and operations a pass cannot do without, and `exact(case, seed)` the floating-point results in 64 bits where they
can be had directly.

Node arrays are sized for the worst case and a build writes the nodes it makes, so they start as zeros here.
"""
import math

import numpy as np
import torch

from cudart_b200 import core, proposal, scenes

FOV = scenes.FOV_60
TEMPORARY = 1 << 24  # elements of one temporary of exact()


def listed():
    return [
        # a viewer of one small terrain, everything at its defaults: rebuild, camera rays, hits, one diffuse bounce (the
        # smallest calls: their time is launches and latency)
        dict(name="frame_terrain_32k", kind="frame", grid=128, width=512, height=512),
        # one deforming mesh of a million triangles, rebuilt with the tree that the fast walks use
        dict(name="build_soup_1m", kind="build", scene="soup", faces=1 << 20, clusters=True, hitbox=False),
        # a large mesh loaded once, with the hit box its file carries left out and node records only
        dict(name="build_soup_16m", kind="build", scene="soup", faces=1 << 24, clusters=False, hitbox=False),
        # many uneven meshes built by one call
        dict(name="batch_build_1024", kind="batch_build", meshes=1024, min_faces=64, max_faces=65536, clusters=True),
        # the sort as a function of its own: 32-bit keys with the values a caller has (an odd count)
        dict(name="sort_pairs_16m", kind="sort", count=(1 << 24) - 5, bits=32, values="given"),
        # a still scene under a moving camera: camera rays, hits, one diffuse bounce per hit
        dict(name="trace_soup_1080p", kind="trace", faces=1 << 20, width=1920, height=1080, walk="clusters"),
        # incoherent rays of many meshes in one call
        dict(name="batch_trace_1024", kind="batch_trace", meshes=1024, min_faces=64, max_faces=65536, min_side=64, max_side=512),
        # the headline frame: 64 deformed instances rebuilt, 33.2M camera rays traced, their bounces traced
        dict(name="frame_instances_64", kind="instances", count=64, scale=0.0625, width=960, height=540),
        # a static mesh's SAH tree
        dict(name="sah_soup_1m", kind="sah", faces=1 << 20, depth=0),
        # the rasteriser on the same mesh
        dict(name="raster_soup_1080p", kind="raster", faces=1 << 20, width=1920, height=1080),
        # the proposal network: slots for two million rays, and one training step (forward, backward, Adam)
        dict(name="propose_2m", kind="propose", rays=(1 << 21) - 77),
        dict(name="train_8192", kind="train", batch=8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "build", "build", "batch_build", "sort", "trace", "trace", "batch_trace", "instances", "sah",
                       "raster", "propose", "train"])
    if kind == "frame":
        return dict(kind=kind, grid=_log_int(rng, 16, 512), width=_log_int(rng, 64, 1024), height=_log_int(rng, 64, 768))
    if kind == "build":
        return dict(kind=kind, scene=rng.choice(["soup", "terrain"]), faces=_log_int(rng, 2000, 12_000_000),
                    clusters=rng.random() < 0.6, hitbox=rng.random() < 0.5)
    if kind == "batch_build":
        return dict(kind=kind, meshes=_log_int(rng, 8, 1024), min_faces=_log_int(rng, 32, 2000), max_faces=_log_int(rng, 4000, 65536),
                    clusters=rng.random() < 0.7)
    if kind == "sort":
        return dict(kind=kind, count=_log_int(rng, 1000, 1 << 24), bits=rng.choice([8, 16, 24, 30, 32, 32, 32]),
                    values=rng.choice(["given", "positions", "none"]))
    if kind == "trace":
        return dict(kind=kind, faces=_log_int(rng, 1 << 14, 1 << 21), width=_log_int(rng, 200, 1920), height=_log_int(rng, 150, 1080),
                    walk=rng.choice(["clusters", "clusters", "default"]))
    if kind == "batch_trace":
        return dict(kind=kind, meshes=_log_int(rng, 8, 700), min_faces=_log_int(rng, 32, 2000), max_faces=_log_int(rng, 4000, 65536),
                    min_side=_log_int(rng, 16, 96), max_side=_log_int(rng, 100, 400))
    if kind == "instances":
        return dict(kind=kind, count=_log_int(rng, 4, 60), scale=1.0 / _log_int(rng, 16, 256), width=8 * rng.randint(20, 120),
                    height=4 * rng.randint(30, 135))
    if kind == "sah":
        return dict(kind=kind, faces=_log_int(rng, 4000, 1 << 20), depth=rng.choice([0, 0, 6, 12]))
    if kind == "raster":
        return dict(kind=kind, faces=_log_int(rng, 4000, 1 << 20), width=_log_int(rng, 200, 1920), height=_log_int(rng, 150, 1080))
    if kind == "propose":
        return dict(kind=kind, rays=_log_int(rng, 5000, 1 << 21))
    return dict(kind="train", batch=128 * _log_int(rng, 2, 64))


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _soup(n, g):
    """n triangles, centroids uniform in the unit cube, corners moved by N(0, 0.01^2) (scenes.soup, on the device)."""
    c = torch.rand((n, 1, 3), generator=g, device="cuda")
    v = torch.zeros((n, 3, 4), device="cuda")
    v[:, :, :3] = torch.randn((n, 3, 3), generator=g, device="cuda").mul_(0.01).add_(c)
    f = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    f[:, :3] = torch.arange(3 * n, dtype=torch.int32, device="cuda").view(n, 3)
    return v.view(3 * n, 4), f


def _terrain(grid, seed):
    """A height field over grid x grid vertices (scenes.terrain, on the device)."""
    rng = np.random.default_rng(seed)
    fr, phi, th = rng.uniform(1.0, 8.0, 4), rng.uniform(0.0, 2.0 * math.pi, 4), rng.uniform(0.0, 2.0 * math.pi, 4)
    xs = torch.linspace(-1.0, 1.0, grid, dtype=torch.float64, device="cuda")
    x, z = xs.view(1, grid), xs.view(grid, 1)
    y = sum(torch.sin(fr[k] * (math.cos(th[k]) * x + math.sin(th[k]) * z) + phi[k]) for k in range(4)) * 0.1
    v = torch.zeros((grid, grid, 4), device="cuda")
    v[:, :, 0], v[:, :, 1], v[:, :, 2] = x, y, z
    i = torch.arange(grid - 1, dtype=torch.int32, device="cuda")
    a = (i.view(-1, 1) * grid + i.view(1, -1)).reshape(-1)
    f = torch.zeros((a.numel(), 2, 4), dtype=torch.int32, device="cuda")
    f[:, 0, 0], f[:, 0, 1], f[:, 0, 2] = a, a + grid, a + 1
    f[:, 1, 0], f[:, 1, 1], f[:, 1, 2] = a + 1, a + grid, a + grid + 1
    return v.view(-1, 4), f.view(-1, 4)


def _grid_of(faces):
    return max(2, int(round(math.sqrt(faces / 2.0))) + 1)


def _mesh(case, seed):
    if case["scene"] == "terrain":
        return _terrain(_grid_of(case["faces"]), seed)
    return _soup(case["faces"], _gen(seed))


def _face_count(case):
    return 2 * (_grid_of(case["faces"]) - 1) ** 2 if case.get("scene") == "terrain" else case["faces"]


def _tree(n, max_nodes):
    """The buffers of a single-mesh build."""
    def i32(*shape):
        return torch.zeros(shape, dtype=torch.int32, device="cuda")
    return core.Tree(nodes=i32(max_nodes, 8), boxes=torch.zeros((n, 8), device="cuda"), indices=i32(n), codes=i32(n), faces=i32(n, 4),
                     tris=torch.zeros((n, 12), device="cuda"), info=i32(8),
                     accel=torch.zeros(core.accel_bytes(n), dtype=torch.uint8, device="cuda"))


def _tree_out(t):
    return dict(nodes=t.nodes, boxes=t.boxes, indices=t.indices, codes=t.codes, faces=t.faces, tris=t.tris, info=t.info)


def _hits(h):
    return dict(id=h["id"], t=h["t"], uv=h["uv"])


def _hit_buffers(rays):
    return dict(id=torch.zeros(rays, dtype=torch.int32, device="cuda"), t=torch.zeros(rays, device="cuda"),
                uv=torch.zeros((rays, 2), device="cuda"), err=torch.zeros(1, dtype=torch.int32, device="cuda"))


def _ray_buffers(rays):
    return torch.zeros((rays, 4), device="cuda"), torch.zeros((rays, 4), device="cuda")


def _batch_sizes(case):
    """(faces, terrain or not) per mesh: the same for every seed, whose meshes differ in shape alone."""
    rng = np.random.default_rng(case["meshes"])
    lo, hi = math.log(case["min_faces"]), math.log(case["max_faces"])
    return [(int(round(math.exp(rng.uniform(lo, hi)))), rng.random() < 0.5) for _ in range(case["meshes"])]


def _batch(case, seed):
    """Uneven meshes, terrain or soup by a fair coin (scenes.batch_meshes, on the device)."""
    g = _gen(seed)
    verts, faces, fo, vo, terrain = [], [], [0], [0], []
    for i, (n, is_terrain) in enumerate(_batch_sizes(case)):
        v, f = _terrain(_grid_of(n), 1000 * seed + i) if is_terrain else _soup(n, g)
        verts.append(v)
        faces.append(f)
        fo.append(fo[-1] + f.shape[0])
        vo.append(vo[-1] + v.shape[0])
        terrain.append(is_terrain)
    return torch.cat(verts), torch.cat(faces), fo, vo, terrain


def _batch_out(t):
    return dict(nodes=t.nodes, boxes=t.boxes, indices=t.indices, codes=t.codes, faces=t.faces, tris=t.tris, info=t.info)


def _view(case):
    """Where the camera is and what it looks at."""
    return ((0.0, 1.5, -2.5), (0.0, 0.0, 0.0)) if case["kind"] == "frame" else ((0.5, 0.5, -0.4), (0.5, 0.5, 0.5))


def _jittered(seed, center):
    rng = np.random.default_rng(seed)
    return [x + 0.02 * float(rng.uniform(-1, 1)) for x in center]


def _camera(seed, center, target, width, height):
    return core.make_camera(_jittered(seed, center), target, fov=FOV, ratio=float(np.float32(width) / np.float32(height)))


def _rays_in_box(n, g, lo, hi):
    o, d = _ray_buffers(n)
    lo, hi = torch.tensor(lo, device="cuda"), torch.tensor(hi, device="cuda")
    o[:, :3] = lo + (hi - lo) * torch.rand((n, 3), generator=g, device="cuda")
    v = torch.randn((n, 3), generator=g, device="cuda")
    d[:, :3] = v / v.norm(dim=1, keepdim=True).clamp(min=1e-20)
    return o, d


PROPOSE_BOX = (-1.5, -0.6, -1.5, 1.5, 1.4, 1.5)


# ----------------------------------------------------------------------------
# prepare / run
# ----------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "frame":
        s["v"], s["f"] = _terrain(case["grid"], seed)
        s["tree"] = _tree(s["f"].shape[0], 2 * s["f"].shape[0] - 1)
        s["camera"] = _camera(seed, *_view(case), case["width"], case["height"])
        rays = case["width"] * case["height"]
        s.update(rays=_ray_buffers(rays), bounce=_ray_buffers(rays) + (torch.zeros(rays, device="cuda"),), h1=_hit_buffers(rays),
                 h2=_hit_buffers(rays), seed=seed)
    elif kind in ("build", "sah"):
        s["v"], s["f"] = _mesh(dict(case, scene=case.get("scene", "soup")), seed)
        n = s["f"].shape[0]
        s["tree"] = _tree(n, core.sah_sizes(n, case["depth"])[1] if kind == "sah" else 2 * n - 1)
        s["hitbox"] = torch.cat([s["v"].amin(0), s["v"].amax(0)]).tolist() if case.get("hitbox") else None
    elif kind == "batch_build":
        s["v"], s["f"], s["fo"], s["vo"], _ = _batch(case, seed)
        s["tree"] = core.batch_build(s["v"], s["f"], s["fo"], s["vo"], clusters=case["clusters"])
        s["tree"].nodes.zero_()
    elif kind == "sort":
        g = _gen(seed)
        n = case["count"]
        s["keys"] = torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device="cuda").to(torch.int32)
        if case["bits"] < 32:
            s["keys"].bitwise_and_((1 << case["bits"]) - 1)
        s["values"] = torch.randint(0, 1 << 31, (n,), generator=g, device="cuda").to(torch.int32) if case["values"] == "given" else None
        s["k"], s["w"] = torch.zeros_like(s["keys"]), torch.zeros_like(s["keys"])
    elif kind == "trace":
        v, f = _soup(case["faces"], _gen(seed))
        s["tree"] = core.build_lbvh(v, f, clusters=case["walk"] == "clusters")
        s["camera"] = _camera(seed, *_view(case), case["width"], case["height"])
        rays = case["width"] * case["height"]
        s.update(rays=_ray_buffers(rays), bounce=_ray_buffers(rays) + (torch.zeros(rays, device="cuda"),), h1=_hit_buffers(rays),
                 h2=_hit_buffers(rays), seed=seed)
        s["first"] = s["second"] = None  # the default walk
        if case["walk"] == "clusters":  # packets over pixel tiles, refilled warps for the bounces
            s["first"] = dict(clusters=True, image_width=case["width"], persistent=True, blocks_per_sm=16, packet=True)
            s["second"] = dict(clusters=True, persistent=True, blocks_per_sm=8, refill=True, lane_threshold=8)
    elif kind == "batch_trace":
        v, f, fo, vo, terrain = _batch(case, seed)
        s["tree"] = core.batch_build(v, f, fo, vo, clusters=True)
        rng = np.random.default_rng(case["meshes"])
        side = np.exp(rng.uniform(math.log(case["min_side"]), math.log(case["max_side"]), case["meshes"])).astype(np.int64)
        off = np.concatenate([[0], np.cumsum(side * side)])
        rays = int(off[-1])
        g = _gen(seed)
        which = torch.repeat_interleave(torch.arange(case["meshes"], device="cuda"), torch.from_numpy(side * side).cuda())
        t = torch.tensor(terrain, device="cuda")[which].unsqueeze(1)
        mid, rad = torch.where(t, 0.0, 0.5), torch.where(t, 1.5, 0.92)  # spheres around a terrain and around the unit cube
        p, q = (torch.nn.functional.normalize(torch.randn((rays, 3), generator=g, device="cuda")) for _ in range(2))
        q = q * torch.rand((rays, 1), generator=g, device="cuda").pow(1.0 / 3.0)
        o, d = _ray_buffers(rays)
        o[:, :3] = mid + rad * p
        d[:, :3] = rad * (q - p)
        s.update(rays=(o, d), off=torch.from_numpy(off).to(torch.int32).cuda(), h1=_hit_buffers(rays),
                 first=dict(clusters=True, persistent=True, blocks_per_sm=8, refill=True, lane_threshold=8))
    elif kind == "instances":
        n, w, h = case["count"], case["width"], case["height"]
        base = scenes.learned_scene(case["scale"])
        s["v"] = scenes.displace_instances(torch.from_numpy(base.vertices).cuda(), n, 0, seed=seed)
        s["f"] = torch.from_numpy(base.faces.view(np.int32)).cuda().repeat(n, 1).contiguous()
        s["fo"] = [i * base.face_count for i in range(n + 1)]
        s["vo"] = [i * base.vertex_count for i in range(n + 1)]
        cams = [core.make_camera(c.center, c.target, fov=c.fov, ratio=c.ratio) for c in scenes.instance_cameras(n, w, h)]
        s["bases"] = core.camera_bases(cams, w, h)
        s["tree"] = core.batch_build(s["v"], s["f"], s["fo"], s["vo"], clusters=True)
        s["tree"].nodes.zero_()
        rays = n * w * h
        s.update(rays=_ray_buffers(rays), bounce=_ray_buffers(rays) + (torch.zeros(rays, device="cuda"),), h1=_hit_buffers(rays),
                 h2=_hit_buffers(rays), off=torch.tensor([i * w * h for i in range(n + 1)], dtype=torch.int32, device="cuda"), seed=seed)
        s["first"] = dict(clusters=True, persistent=True, blocks_per_sm=16, packet=True, tiles=[n, w, h])
        s["second"] = dict(clusters=True, persistent=True, blocks_per_sm=8, refill=True, lane_threshold=8)
    elif kind == "raster":
        s["v"], s["f"] = _soup(case["faces"], _gen(seed))
        target = (0.5, 0.5, 0.5)
        cam = _camera(seed, (0.55, 0.6, -0.4), target, case["width"], case["height"])
        s["matrix"] = core.raster_matrix(cam, target)
    elif kind == "propose":
        s["net"] = proposal.ProposalNet(seed=seed)
        s["rays"] = _rays_in_box(case["rays"], _gen(seed), PROPOSE_BOX[:3], PROPOSE_BOX[3:])
        s["out"] = torch.zeros(case["rays"], dtype=torch.int32, device="cuda")
    else:
        s["net"] = proposal.ProposalNet(seed=seed)
        s["rays"], s["labels"] = _train_batch(case, seed)
    return s


def _train_batch(case, seed):
    """Rays and a label per ray: the cell (of 16 x 16 x 16) that holds a point further along it."""
    o, d = _rays_in_box(case["batch"], _gen(seed), PROPOSE_BOX[:3], PROPOSE_BOX[3:])
    p = (o + 0.5 * d)[:, :3]
    lo, hi = torch.tensor(PROPOSE_BOX[:3], device="cuda") - 0.5, torch.tensor(PROPOSE_BOX[3:], device="cuda") + 0.5
    q = ((p - lo) / (hi - lo) * 16).clamp(0, 15).to(torch.int32)
    return (o, d), (q[:, 0] * 256 + q[:, 1] * 16 + q[:, 2]).contiguous()


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("frame", "trace"):
        if kind == "frame":
            core.build_lbvh(s["v"], s["f"], out=s["tree"])
        first, second = s.get("first"), s.get("second")
        o, d = core.primary_rays(s["camera"], case["width"], case["height"], out=s["rays"])
        h1 = core.trace(s["tree"], o, d, out=s["h1"], schedule=first)
        b = core.bounce_rays(s["tree"].tris, o, d, h1["id"], h1["t"], s["seed"], out=s["bounce"])
        h2 = core.trace(s["tree"], b[0], b[1], tmax=b[2], out=s["h2"], schedule=second)
        out = dict(h1=_hits(h1), h2=_hits(h2), orig=o, dir=d, bounce_orig=b[0], bounce_dir=b[1], bounce_tmax=b[2])
        return dict(out, tree=_tree_out(s["tree"])) if kind == "frame" else out
    if kind == "build":
        return _tree_out(core.build_lbvh(s["v"], s["f"], hitbox=s["hitbox"], out=s["tree"], clusters=case["clusters"]))
    if kind == "sah":
        t = _tree_out(core.build_sah(s["v"], s["f"], lbvh_depth=case["depth"], out=s["tree"]))
        t.pop("codes")
        return t
    if kind == "batch_build":
        return _batch_out(core.batch_build(s["v"], s["f"], s["fo"], s["vo"], out=s["tree"], clusters=case["clusters"]))
    if kind == "sort":
        s["k"].copy_(s["keys"])  # the sort works in place: a program's new keys arrive in its buffer
        if case["values"] == "none":
            return core.sort_keys(s["k"], case["bits"])
        if case["values"] == "given":
            s["w"].copy_(s["values"])
        return core.sort_pairs(s["k"], s["w"], case["bits"], init_values=case["values"] == "positions")
    if kind == "batch_trace":
        return _hits(core.batch_trace(s["tree"], s["rays"][0], s["rays"][1], s["off"], out=s["h1"], schedule=s["first"]))
    if kind == "instances":
        tree = core.batch_build(s["v"], s["f"], s["fo"], s["vo"], out=s["tree"], clusters=True)
        o, d = core.batch_primary_rays(s["bases"], case["width"], case["height"], out=s["rays"])
        h1 = core.batch_trace(tree, o, d, s["off"], out=s["h1"], schedule=s["first"], bounce=(s["seed"], s["bounce"]))
        b = h1["b"]
        h2 = core.batch_trace(tree, b[0], b[1], s["off"], tmax=b[2], out=s["h2"], schedule=s["second"])
        return dict(h1=_hits(h1), h2=_hits(h2), bounce_orig=b[0], bounce_dir=b[1], bounce_tmax=b[2], nodes=tree.nodes,
                    indices=tree.indices, info=tree.info)
    if kind == "raster":
        r = core.rasterize(s["v"], s["f"], s["matrix"], case["width"], case["height"])
        return dict(id=r["id"], uv=r["uv"], depth=r["depth"])
    net = s["net"]
    if kind == "propose":
        return net.propose(s["rays"][0], s["rays"][1], PROPOSE_BOX, out=s["out"])
    loss = net.train_step(s["rays"][0], s["rays"][1], s["labels"], PROPOSE_BOX)
    return dict(loss=loss, grads=list(net.grads), weights=list(net.params))


# ----------------------------------------------------------------------------
# work
# ----------------------------------------------------------------------------
def _build_bytes(verts, faces):
    # vertices and faces in; boxes, indices, codes, reordered faces and triangles out; a node of 32 bytes per 50 faces or so
    return 16 * verts + faces * (16 + 32 + 4 + 4 + 16 + 48 + 32 * 0.02)


def _mean_log_uniform(lo, hi):
    return (hi - lo) / math.log(hi / lo) if hi > lo else float(lo)


def work(case):
    kind = case["kind"]
    macs = 144 * 128 + 2 * 128 * 128 + 128 * 4096  # the proposal network, per ray
    if kind == "frame":
        n, v, r = 2 * (case["grid"] - 1) ** 2, case["grid"] ** 2, case["width"] * case["height"]
        return dict(bytes=_build_bytes(v, n) + 2 * (48 * n + 48 * r) + 36 * r, flops=0)
    if kind in ("build", "sah"):
        n = _face_count(case)
        return dict(bytes=_build_bytes(_grid_of(case["faces"]) ** 2 if case.get("scene") == "terrain" else 3 * n, n), flops=0)
    if kind == "batch_build":
        n = case["meshes"] * _mean_log_uniform(case["min_faces"], case["max_faces"])
        return dict(bytes=_build_bytes(1.75 * n, n), flops=0)
    if kind == "sort":
        return dict(bytes=case["count"] * (8 + {"given": 8, "positions": 4, "none": 0}[case["values"]]), flops=0)
    if kind == "trace":
        r = case["width"] * case["height"]
        return dict(bytes=2 * (48 * case["faces"] + 48 * r) + 36 * r, flops=0)
    if kind == "batch_trace":
        n = case["meshes"] * _mean_log_uniform(case["min_faces"], case["max_faces"])
        lo, hi = case["min_side"], case["max_side"]
        r = case["meshes"] * ((hi * hi - lo * lo) / (2 * math.log(hi / lo)) if hi > lo else lo * lo)
        return dict(bytes=48 * n + 48 * r, flops=0)
    if kind == "instances":
        n, r = case["count"] * case["scale"] * 4_022_242, case["count"] * case["width"] * case["height"]
        return dict(bytes=_build_bytes(2.7 * n, n) + 2 * (48 * n + 48 * r) + 36 * r, flops=0)
    if kind == "raster":
        return dict(bytes=64 * case["faces"] + 16 * case["width"] * case["height"], flops=0)
    if kind == "propose":
        return dict(bytes=36 * case["rays"] + 2 * 579_968, flops=2 * macs * case["rays"])
    return dict(bytes=36 * case["batch"] + 579_968 * (4 * 7 + 2), flops=6 * macs * case["batch"])


# ----------------------------------------------------------------------------
# exact
# ----------------------------------------------------------------------------
def _boxes64(v, f):
    p = v[:, :3].double()[f[:, :3].long()]
    out = torch.zeros((f.shape[0], 8), dtype=torch.float64, device="cuda")
    out[:, :3], out[:, 4:7] = p.amin(1), p.amax(1)
    return out


def _pinhole64(center, target, width, height):
    """Camera rays in 64 bits: a camera at center looking at target without roll, rows from the top left."""
    c, t = np.array(center, np.float32).astype(np.float64), np.array(target, np.float64)
    d = (t - c) / np.linalg.norm(t - c)
    side = np.cross(d, [0.0, 1.0, 0.0])
    side /= np.linalg.norm(side)
    up = np.cross(side, d)
    y = math.tan(0.5 * FOV)
    x = y * width / height
    i = torch.arange(width * height, device="cuda")
    px, py = (i % width).double().unsqueeze(1), torch.div(i, width, rounding_mode="floor").double().unsqueeze(1)
    side, up, d = (torch.tensor(a, device="cuda") for a in (side, up, d))
    orig, dirs = (torch.zeros((width * height, 4), dtype=torch.float64, device="cuda") for _ in range(2))
    orig[:, :3] = torch.tensor(c, device="cuda")
    dirs[:, :3] = (up * y + side * x + d) - px * (side * (2 * x / width)) - py * (up * (2 * y / height))
    return orig, dirs


def _closest64(v, f, orig, dirs):
    """Closest hits in 64 bits, every ray against every triangle (Moeller-Trumbore; determinants below 1e-6 miss)."""
    p = v[:, :3].double()[f[:, :3].long()]
    v0, e1, e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    rays, faces = orig.shape[0], f.shape[0]
    best = torch.full((rays,), float(np.float32(core.HUGE)), dtype=torch.float64, device="cuda")
    uv = torch.zeros((rays, 2), dtype=torch.float64, device="cuda")
    step = max(1, TEMPORARY // faces)

    def cross(a, b):
        return (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])

    def dot(a, b):
        return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]

    a, e, g = ([x[:, k].unsqueeze(0) for k in range(3)] for x in (v0, e1, e2))
    for r in range(0, rays, step):
        o, d = ([x[r:r + step, k].unsqueeze(1) for k in range(3)] for x in (orig, dirs))
        pv = cross(d, g)
        det = dot(e, pv)
        tv = [o[k] - a[k] for k in range(3)]
        q = cross(tv, e)
        u, w, t = dot(tv, pv) / det, dot(d, q) / det, dot(g, q) / det
        ok = (det.abs() >= 1e-6) & (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 0)
        t, k = torch.where(ok, t, math.inf).min(1)
        hit = t < best[r:r + step]
        best[r:r + step] = torch.where(hit, t, best[r:r + step])
        at = torch.stack([x.gather(1, k.unsqueeze(1)).squeeze(1) for x in (u, w)], 1)
        uv[r:r + step] = torch.where(hit.unsqueeze(1), at, 0.0)
    return dict(id=None, t=best, uv=uv)


def _exact_train(case, seed):
    """One training step in 64 bits: sin/cos features, three ReLU layers, softmax cross-entropy, Adam's first step."""
    (o, d), labels = _train_batch(case, seed)
    params = [p.double().requires_grad_(True) for p in proposal.ProposalNet(seed=seed).params]
    lo, hi = (torch.tensor(b, dtype=torch.float64, device="cuda") for b in (PROPOSE_BOX[:3], PROPOSE_BOX[3:]))
    u = torch.cat([(o[:, :3].double() - lo) / (hi - lo) * 2 - 1, torch.nn.functional.normalize(d[:, :3].double())], 1)
    angle = (math.pi * u.unsqueeze(2) * 2.0 ** torch.arange(12, dtype=torch.float64, device="cuda"))
    x = torch.zeros((case["batch"], 192), dtype=torch.float64, device="cuda")
    x[:, :144] = torch.stack([torch.sin(angle), torch.cos(angle)], 3).flatten(1)
    for layer in range(3):
        x = torch.relu(x @ params[2 * layer].t() + params[2 * layer + 1])
    loss = torch.nn.functional.cross_entropy(x @ params[6].t() + params[7], labels.long())
    loss.backward()
    grads = [p.grad for p in params]
    weights = [p.detach() - 1e-3 * g / (g.abs() + 1e-8) for p, g in zip(params, grads)]  # m and v divide to the gradient itself
    return dict(loss=loss.detach().reshape(1), grads=grads, weights=weights)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("build", "sah"):
        v, f = _mesh(dict(case, scene=case.get("scene", "soup")), seed)
        out = dict(nodes=None, boxes=_boxes64(v, f), indices=None, codes=None, faces=None, tris=None, info=None)
        if kind == "sah":
            out.pop("codes")
        return out
    if kind == "batch_build":
        v, f, fo, vo, _ = _batch(case, seed)
        base = torch.repeat_interleave(torch.tensor(vo[:-1], device="cuda"), torch.tensor(fo, device="cuda").diff())
        g = f.clone()
        g[:, :3] += base.to(torch.int32).unsqueeze(1)
        return dict(nodes=None, boxes=_boxes64(v, g), indices=None, codes=None, faces=None, tris=None, info=None)
    if kind in ("frame", "trace"):  # the bounces are drawn at random from the hits
        v, f = _terrain(case["grid"], seed) if kind == "frame" else _soup(case["faces"], _gen(seed))
        center, target = _view(case)
        orig, dirs = _pinhole64(_jittered(seed, center), target, case["width"], case["height"])
        few = f.shape[0] * orig.shape[0] <= 40_000_000_000
        out = dict(h1=_closest64(v, f, orig, dirs) if few else None, h2=None, orig=orig, dir=dirs, bounce_orig=None, bounce_dir=None,
                   bounce_tmax=None)
        if kind == "frame":
            out["tree"] = dict(nodes=None, boxes=_boxes64(v, f), indices=None, codes=None, faces=None, tris=None, info=None)
        return out
    if kind == "train":
        return _exact_train(case, seed)
    return None
