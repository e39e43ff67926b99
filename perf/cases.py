"""The work that programs have the path-tracing pass do, as cases that can be timed and compared.

Every case goes through the C ABI of include/bsm_pt.h (bound by the package's ctypes mirror): frames rendered
into device memory, batches of views, requests to the serving loop, instances that move between frames, rays
traced by the stage entry points, primary-hit outputs, frames with the radiance cache, and BVH rebuilds.
Scenes are the repository's own procedural ones at the sizes its tests, benchmark and serving mix use.  The
contexts and the scenes are made once per process and stay resident, as in a renderer; cameras, seeds, rays,
transforms and rebuilt meshes come from the case's seed.
"""
import ctypes as C
import importlib
import math
import random

import numpy as np
import torch

bsm = importlib.import_module("bisemutum-engine_gb300")

# name -> (generator kind, terrain vertices per side, spheres, triangles)
SCENES = {
    "room": (bsm.BSM_SCENE_ROOM, 0, 64, 20504),
    "terrain_250k": (bsm.BSM_SCENE_TERRAIN, 256, 250, 250050),
    "terrain_1.5m": (bsm.BSM_SCENE_TERRAIN, 512, 2000, 1482242),
    "terrain_5m": (bsm.BSM_SCENE_TERRAIN, 1024, 6000, 4973058),
}


def listed():
    return [
        # the smallest call: a thumbnail or an editor's preview while a slider moves
        {"name": "preview_room", "kind": "render", "scene": "room", "width": 128, "height": 128, "spp": 1,
         "segments": 4, "deterministic": False, "jitter": False},
        # a small converged image, bit-reproducible (regression images, caches of thumbnails)
        {"name": "room_256_reproducible", "kind": "render", "scene": "room", "width": 256, "height": 256, "spp": 16,
         "segments": 4, "deterministic": True, "jitter": False},
        # one progressive 1-spp frame at full resolution: what the engine's renderer asks for every frame
        {"name": "frame_1spp_1080p", "kind": "render", "scene": "terrain_1.5m", "width": 1920, "height": 1080,
         "spp": 1, "segments": 8, "deterministic": False, "jitter": False},
        # a final frame: the largest single call of the benchmark
        {"name": "frame_64spp_1080p", "kind": "render", "scene": "terrain_1.5m", "width": 1920, "height": 1080,
         "spp": 64, "segments": 8, "deterministic": False, "jitter": False},
        # many views of odd sizes and sample counts in one call (light probes, turntables, data sets)
        {"name": "batch_uneven_views", "kind": "batch", "scene": "terrain_250k", "views": 12, "min_side": 65,
         "max_side": 517, "max_spp": 16, "segments": 8},
        # requests of several users to the serving loop, submitted together and waited for
        {"name": "serve_mixed_requests", "kind": "serve", "requests": 16, "max_width": 960, "max_spp": 8,
         "segments": 8},
        # an animated two-level scene: new transforms, then a preview frame
        {"name": "moving_instances", "kind": "moving", "instances": 1000, "ground": 128, "width": 641, "height": 359,
         "spp": 1, "segments": 4},
        # baking: closest hits and occlusion of many incoherent rays of a large scene
        {"name": "trace_rays_1m", "kind": "trace", "scene": "terrain_1.5m", "rays": 1000003},
        # a script's or editor's visibility queries: few rays, small scene
        {"name": "trace_rays_2k", "kind": "trace", "scene": "room", "rays": 2047},
        # depth, G-buffer and hit positions of a frame, which the engine's other passes read
        {"name": "primary_1080p", "kind": "primary", "scene": "terrain_1.5m", "width": 1920, "height": 1080},
        # a real-time frame with the learned radiance cache, its online training included
        {"name": "cached_frame_720p", "kind": "cached", "scene": "terrain_1.5m", "width": 1280, "height": 720,
         "spp": 1, "train": True},
        # an edited or streamed mesh: the BVH rebuilt, then rays traced through the new tree
        {"name": "rebuild_1.5m", "kind": "rebuild", "scene": "terrain_1.5m", "rays": 65536},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "batch", "serve", "moving", "trace", "trace", "primary",
                       "cached", "rebuild"])
    scene = rng.choice(["room", "terrain_250k", "terrain_1.5m", "terrain_5m"])
    width = _log_int(rng, 96, 1920)
    height = max(33, int(width * rng.uniform(0.45, 0.75)))
    if kind == "render":
        spp = rng.choice([1, 1, 2, 4, 7, 16, 32])
        return {"kind": kind, "scene": scene, "width": width, "height": height, "spp": spp,
                "segments": rng.choice([2, 4, 8]), "deterministic": rng.random() < 0.3, "jitter": rng.random() < 0.4}
    if kind == "batch":
        return {"kind": kind, "scene": scene, "views": rng.randint(2, 24), "min_side": rng.randint(33, 128),
                "max_side": rng.randint(200, 700), "max_spp": rng.choice([4, 16, 32]),
                "segments": rng.choice([2, 4, 8])}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(2, 32), "max_width": _log_int(rng, 200, 1920),
                "max_spp": rng.choice([4, 16]), "segments": rng.choice([4, 8])}
    if kind == "moving":
        return {"kind": kind, "instances": _log_int(rng, 50, 4000), "ground": rng.choice([64, 128, 192]),
                "width": width, "height": height, "spp": rng.choice([1, 2, 4]), "segments": rng.choice([2, 4, 8])}
    if kind == "trace":
        return {"kind": kind, "scene": scene, "rays": _log_int(rng, 100, 4000000)}
    if kind == "primary":
        return {"kind": kind, "scene": scene, "width": width, "height": height}
    if kind == "cached":
        return {"kind": kind, "scene": rng.choice(["room", "terrain_250k", "terrain_1.5m"]), "width": width,
                "height": height, "spp": rng.choice([1, 2, 4]), "train": rng.random() < 0.7}
    return {"kind": kind, "scene": rng.choice(["room", "terrain_250k", "terrain_1.5m"]),
            "rays": _log_int(rng, 1000, 200000)}


# ------------------------------------------------------------ resident things ----
_contexts = {}    # role -> Context
_meshes = {}      # scene name -> SceneData
_resident = {}    # (role, scene name) -> scene id


def _context(role="main"):
    if role not in _contexts:
        _contexts[role] = bsm.Context(0)
    return _contexts[role]


def _mesh(name, seed=1):
    kind, grid, spheres, _ = SCENES[name]
    if seed != 1:
        return bsm.generate_scene(kind, seed=seed, grid=grid, spheres=spheres)
    if name not in _meshes:
        _meshes[name] = bsm.generate_scene(kind, seed=1, grid=grid, spheres=spheres)
    return _meshes[name]


def _scene(name, role="main"):
    if (role, name) not in _resident:
        _resident[role, name] = _context(role).load_scene(_mesh(name))
    return _resident[role, name]


def _camera(mesh, rng, width, height):
    """The scene's own camera, moved and turned a little."""
    base = mesh.camera
    extent = float(np.max(mesh.positions.max(0) - mesh.positions.min(0)))
    pos = [p + rng.uniform(-0.02, 0.02) * extent for p in base.position]
    front = [f + rng.uniform(-0.05, 0.05) for f in base.front]
    return bsm.make_camera(pos, front, yfov_deg=float(base.yfov_deg), width=width, height=height)


def _device_view(image):
    return bsm.ViewOutput(image.data_ptr(), 0, bsm.BSM_DEVICE)


def _rays(mesh, n, seed):
    """Half of the rays leave points of the surface into the hemisphere above (occlusion bakes, probes), half
    start anywhere in the scene's box in any direction."""
    rng = np.random.default_rng(seed)
    lo, hi = mesh.positions.min(0), mesh.positions.max(0)
    extent = float((hi - lo).max())
    rays = np.zeros((n, 8), np.float32)
    half = n // 2
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[:half, 1] = np.abs(d[:half, 1])
    rays[:half, 0:3] = mesh.positions[rng.integers(0, len(mesh.positions), half)]
    rays[:half, 1] += 1e-4 * extent
    rays[half:, 0:3] = lo + (hi - lo) * rng.uniform(0.02, 0.98, (n - half, 3))
    rays[:, 4:7] = d
    rays[:, 7] = 4.0 * extent
    return rays


# -------------------------------------------------------------------- states ----
class _State:
    """What a program holds between calls; gives back what it made for itself alone."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        if getattr(self, "cache", None) is not None:
            self.cache.close()
        if getattr(self, "own_scene", None) is not None:
            self.ctx.release(self.own_scene)


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed, random.Random(seed))


def run(state):
    return _RUN[state.kind](state)


def _image(width, height):
    return torch.empty((height, width, 4), dtype=torch.float32, device="cuda")


def _prepare_render(case, seed, rng):
    ctx, sid = _context(), _scene(case["scene"])
    cam = _camera(_mesh(case["scene"]), rng, case["width"], case["height"])
    flags = (bsm.BSM_PT_DETERMINISTIC if case["deterministic"] else 0) | (bsm.BSM_PT_JITTER if case["jitter"] else 0)
    image = _image(case["width"], case["height"])
    return _State(kind="render", ctx=ctx, sid=sid, cam=cam, image=image, out=_device_view(image),
                  settings=bsm.settings(spp=case["spp"], max_segments=case["segments"], seed=seed + 1, flags=flags))


def _run_render(s):
    s.ctx.check(bsm.lib().bsm_render(s.ctx.h, s.sid, C.byref(s.cam), 1, C.byref(s.settings), C.byref(s.out), None))
    return {"image": s.image}


def _prepare_batch(case, seed, rng):
    ctx, sid, mesh = _context(), _scene(case["scene"]), _mesh(case["scene"])
    n = case["views"]
    shape = random.Random(n)   # sizes and sample counts belong to the case, cameras and seeds to the inputs
    views, outs, images = (bsm.ViewDesc * n)(), (bsm.ViewOutput * n)(), []
    for i in range(n):
        side = _log_int(shape, case["min_side"], case["max_side"])
        views[i].camera = _camera(mesh, rng, side, max(1, int(side * shape.uniform(0.6, 1.0))))
        views[i].spp = shape.choice([k for k in (1, 2, 4, 8, 16, 32) if k <= case["max_spp"]])
        views[i].max_segments = case["segments"]
        views[i].seed = seed + i + 1
        images.append(_image(views[i].camera.width, views[i].camera.height))
        outs[i] = _device_view(images[-1])
    return _State(kind="batch", ctx=ctx, sid=sid, views=views, n=n, outs=outs, images=images,
                  settings=bsm.settings(max_segments=case["segments"], seed=seed + 1))


def _run_batch(s):
    s.ctx.check(bsm.lib().bsm_render_batch(s.ctx.h, s.sid, s.views, s.n, C.byref(s.settings), s.outs, None))
    return s.images


def _prepare_serve(case, seed, rng):
    first = "serve" not in _contexts
    ctx = _context("serve")
    names = ("room", "terrain_250k", "terrain_1.5m")
    ids = [_scene(n, "serve") for n in names]
    if first:
        ctx.server_start()
    shape = random.Random(case["requests"])
    reqs, images = [], []
    for i in range(case["requests"]):
        k = shape.randrange(3)
        width = _log_int(shape, 128, case["max_width"])
        height = max(16, int(width * 0.5625))
        img = np.zeros((height, width, 4), np.float32)
        images.append(img)
        reqs.append(bsm.Request(ids[k], _camera(_mesh(names[k]), rng, width, height),
                                shape.choice([c for c in (1, 4, 16) if c <= case["max_spp"]]),
                                shape.choice([c for c in (2, 4, 8) if c <= case["segments"]]), seed + i + 1,
                                img.ctypes.data))
    return _State(kind="serve", ctx=ctx, reqs=reqs, images=images)


def _run_serve(s):
    lib, rids = bsm.lib(), []
    for r in s.reqs:
        rid = C.c_uint64()
        s.ctx.check(lib.bsm_server_submit(s.ctx.h, C.byref(r), C.byref(rid)))
        rids.append(rid)
    status = bsm.RequestStatus()
    for rid in rids:
        s.ctx.check(lib.bsm_server_wait(s.ctx.h, rid, 0, C.byref(status)))
    return s.images


def _prepare_moving(case, seed, rng):
    ctx = _context()
    key = ("main", "instances", case["instances"], case["ground"])
    name = key[1:]
    if name not in _meshes:
        _meshes[name] = bsm.generate_instanced_scene(seed=1, instances=case["instances"], ground=case["ground"])
        _resident[key] = ctx.load_instanced(_meshes[name])
    scene = _meshes[name]
    xf = np.array(scene.inst_transform, np.float32).reshape(-1, 12).copy()
    g = np.random.default_rng(seed)
    xf[1:, [3, 7, 11]] += g.uniform(-0.1, 0.1, (len(xf) - 1, 3)).astype(np.float32)   # the ground stays
    base = scene.camera
    cam = bsm.make_camera([p + rng.uniform(-0.1, 0.1) for p in base.position], list(base.front),
                          yfov_deg=float(base.yfov_deg), width=case["width"], height=case["height"])
    image = _image(case["width"], case["height"])
    return _State(kind="moving", ctx=ctx, sid=_resident[key], xf=np.ascontiguousarray(xf), cam=cam, image=image,
                  out=_device_view(image),
                  settings=bsm.settings(spp=case["spp"], max_segments=case["segments"], seed=seed + 1))


def _run_moving(s):
    s.ctx.update_instances(s.sid, s.xf)
    return _run_render(s)


def _hit_buffers(n):
    return torch.empty((n, 4), dtype=torch.int32, device="cuda"), torch.empty(n, dtype=torch.uint8, device="cuda")


def _hits(raw):
    f = raw.view(torch.float32)
    return {"t": f[:, 0], "prim": raw[:, 1], "uv": f[:, 2:4]}


def _prepare_trace(case, seed, rng):
    rays = torch.from_numpy(_rays(_mesh(case["scene"]), case["rays"], seed)).cuda()
    hits, occluded = _hit_buffers(case["rays"])
    return _State(kind="trace", ctx=_context(), sid=_scene(case["scene"]), rays=rays, hits=hits, occluded=occluded)


def _run_trace(s):
    lib, n = bsm.lib(), s.rays.shape[0]
    rays = s.rays.data_ptr()
    s.ctx.check(lib.bsm_trace_closest(s.ctx.h, s.sid, rays, n, s.hits.data_ptr(), bsm.BSM_DEVICE))
    s.ctx.check(lib.bsm_trace_any(s.ctx.h, s.sid, rays, n, s.occluded.data_ptr(), bsm.BSM_DEVICE))
    return {**_hits(s.hits), "occluded": s.occluded}


def _prepare_primary(case, seed, rng):
    w, h = case["width"], case["height"]
    cam = _camera(_mesh(case["scene"]), rng, w, h)
    depth = torch.empty((h, w), dtype=torch.float32, device="cuda")
    gbuffer = torch.empty((4, h, w, 4), dtype=torch.float32, device="cuda")
    points = _image(w, h)
    out = bsm.PrimaryOutput()
    out.depth = depth.data_ptr()
    for k in range(4):
        out.gbuffer[k] = gbuffer[k].data_ptr()
    out.hit_positions = points.data_ptr()
    out.location = bsm.BSM_DEVICE
    return _State(kind="primary", ctx=_context(), sid=_scene(case["scene"]), cam=cam, out=out, depth=depth,
                  gbuffer=gbuffer, points=points, settings=bsm.settings(seed=seed + 1))


def _run_primary(s):
    s.ctx.check(bsm.lib().bsm_render_primary(s.ctx.h, s.sid, C.byref(s.cam), C.byref(s.settings), 0.01, 10000.0,
                                             C.byref(s.out)))
    return {"depth": s.depth, "points": s.points, "gbuffer": s.gbuffer}


def _prepare_cached(case, seed, rng):
    ctx, sid = _context(), _scene(case["scene"])
    image = _image(case["width"], case["height"])
    return _State(kind="cached", ctx=ctx, sid=sid, cam=_camera(_mesh(case["scene"]), rng, case["width"], case["height"]),
                  image=image, out=_device_view(image), cache=bsm.RadianceCache(ctx, seed=seed + 1),
                  cs=bsm.cache_settings() if case["train"] else bsm.cache_settings(train_steps=0),
                  settings=bsm.settings(spp=case["spp"], max_segments=8, seed=seed + 1,
                                        flags=bsm.BSM_PT_DETERMINISTIC))


def _run_cached(s):
    s.ctx.check(bsm.lib().bsm_render_cached(s.ctx.h, s.sid, C.byref(s.cam), C.byref(s.settings), s.cache.h,
                                            C.byref(s.cs), C.byref(s.out), None, None))
    return {"image": s.image, "weights": s.cache.weights()}


def _prepare_rebuild(case, seed, rng):
    ctx = _context()
    mesh = _mesh(case["scene"], seed=seed + 2)   # another mesh of the same size
    rays = torch.from_numpy(_rays(mesh, case["rays"], seed)).cuda()
    hits, _ = _hit_buffers(case["rays"])
    sid = ctx.upload(mesh)
    return _State(kind="rebuild", ctx=ctx, own_scene=sid, rays=rays, hits=hits)


def _run_rebuild(s):
    stats = s.ctx.build_bvh(s.own_scene)
    s.ctx.check(bsm.lib().bsm_trace_closest(s.ctx.h, s.own_scene, s.rays.data_ptr(), s.rays.shape[0],
                                            s.hits.data_ptr(), bsm.BSM_DEVICE))
    return {**_hits(s.hits), "nodes": stats.num_nodes, "depth": stats.max_depth, "cost": stats.sah_cost}


_PREPARE = {"render": _prepare_render, "batch": _prepare_batch, "serve": _prepare_serve, "moving": _prepare_moving,
            "trace": _prepare_trace, "primary": _prepare_primary, "cached": _prepare_cached,
            "rebuild": _prepare_rebuild}
_RUN = {"render": _run_render, "batch": _run_batch, "serve": _run_serve, "moving": _run_moving, "trace": _run_trace,
        "primary": _run_primary, "cached": _run_cached, "rebuild": _run_rebuild}


# ---------------------------------------------------------------------- work ----
# A ray's traversal: about 15 nodes of eight boxes (six slab planes, two operations each, and the comparisons)
# and 6.5 triangles of about 50 operations; an occlusion ray stops after about 60 % of that.  A path of the
# scenes here traces about 0.45 closest-hit rays per segment it may have (at most 2.3) and 0.75 times as many
# occlusion rays, and shading a vertex takes about 500 operations.
_CLOSEST = 15 * 8 * 14 + 6.5 * 50
_OCCLUSION = 0.6 * _CLOSEST


def _scene_bytes(triangles):
    return triangles * 48 + triangles / 8.15 * 80


def _path_flops(segments):
    rays = min(2.3, 1.0 + 0.45 * (segments - 1))
    return rays * (_CLOSEST + 500) + 0.75 * rays * _OCCLUSION


def work(case):
    kind = case["kind"]
    if kind == "batch":
        shape, pixels, paths = random.Random(case["views"]), 0, 0
        for _ in range(case["views"]):
            side = _log_int(shape, case["min_side"], case["max_side"])
            px = side * max(1, int(side * shape.uniform(0.6, 1.0)))
            pixels += px
            paths += px * shape.choice([k for k in (1, 2, 4, 8, 16, 32) if k <= case["max_spp"]])
        return {"bytes": _scene_bytes(SCENES[case["scene"]][3]) + 16 * pixels, "flops": paths * _path_flops(case["segments"])}
    if kind == "serve":
        shape, pixels, flops = random.Random(case["requests"]), 0, 0
        for _ in range(case["requests"]):
            shape.randrange(3)
            width = _log_int(shape, 128, case["max_width"])
            px = width * max(16, int(width * 0.5625))
            spp = shape.choice([c for c in (1, 4, 16) if c <= case["max_spp"]])
            pixels += px
            flops += px * spp * _path_flops(shape.choice([c for c in (2, 4, 8) if c <= case["segments"]]))
        return {"bytes": 16 * pixels, "flops": flops}
    if kind == "moving":
        px = case["width"] * case["height"]
        return {"bytes": 16 * px + case["instances"] * 176, "flops": px * case["spp"] * _path_flops(case["segments"])}
    scene_bytes = _scene_bytes(SCENES[case["scene"]][3])
    if kind == "trace":
        return {"bytes": scene_bytes + case["rays"] * (32 + 16 + 1), "flops": case["rays"] * (_CLOSEST + _OCCLUSION)}
    if kind == "rebuild":
        # vertices and indices in, nodes and leaf triangles out
        return {"bytes": SCENES[case["scene"]][3] * (6 + 12 + 4) + scene_bytes + case["rays"] * 48,
                "flops": case["rays"] * _CLOSEST}
    px = case["width"] * case["height"]
    if kind == "primary":
        return {"bytes": scene_bytes + px * (4 + 64 + 16), "flops": px * _CLOSEST}
    if kind == "cached":
        # three segments, then the network (34,816 operations a query); training: full-length paths of closest
        # hits and four steps of 16,384 samples (about 186,000 operations each)
        train = 32768 * _path_flops(8) + 4 * 16384 * 186000 if case["train"] else 0
        return {"bytes": scene_bytes + 16 * px + 17408 * 16,
                "flops": px * case["spp"] * (_path_flops(3) + 0.3 * 34816) + train}
    return {"bytes": scene_bytes + 16 * px, "flops": px * case["spp"] * _path_flops(case["segments"])}


# --------------------------------------------------------------------- exact ----
_EXACT_TESTS = 3e10   # ray-triangle pairs that 64-bit brute force gets through in a few seconds


def _closest_f64(mesh, rays):
    """Closest hits by brute force in 64 bits: (t or tmax, found)."""
    p = torch.from_numpy(mesh.positions.astype(np.float64)).cuda()
    idx = torch.from_numpy(mesh.indices.astype(np.int64)).cuda()
    a, b, c = p[idx[:, 0]], p[idx[:, 1]], p[idx[:, 2]]
    e1, e2 = b - a, c - a
    normal = torch.linalg.cross(e1, e2)
    best = rays[:, 7].clone()
    found = torch.zeros(len(rays), dtype=torch.bool, device="cuda")
    step = max(1, int(4e7 // len(a)))
    for i in range(0, len(rays), step):
        o, d, tmin, tmax = rays[i:i + step, 0:3], rays[i:i + step, 4:7], rays[i:i + step, 3:4], rays[i:i + step, 7:8]
        # scalar triple products from matrix products: det = -d.n, and with m = o x d the two edge functions
        det = -(d @ normal.T)
        m = torch.linalg.cross(o, d)
        num_t = o @ normal.T - (a * normal).sum(1)
        u = m @ e2.T + d @ torch.linalg.cross(a, e2).T
        v = -(m @ e1.T + d @ torch.linalg.cross(a, e1).T)
        t = num_t / det
        u, v = u / det, v / det
        hit = (u >= 0) & (v >= 0) & (u + v <= 1) & (t > tmin) & (t <= tmax)
        t = torch.where(hit, t, torch.inf).min(1).values
        found[i:i + step] = torch.isfinite(t)
        best[i:i + step] = torch.where(torch.isfinite(t), t, best[i:i + step])
    return best, found


def exact(case, seed):
    if case["kind"] == "trace" and case["rays"] * SCENES[case["scene"]][3] <= _EXACT_TESTS:
        mesh = _mesh(case["scene"])
        t, _ = _closest_f64(mesh, torch.from_numpy(_rays(mesh, case["rays"], seed)).cuda().double())
        return {"t": t, "prim": None, "uv": None, "occluded": None}
    if case["kind"] == "rebuild" and case["rays"] * SCENES[case["scene"]][3] <= _EXACT_TESTS:
        mesh = _mesh(case["scene"], seed=seed + 2)
        t, _ = _closest_f64(mesh, torch.from_numpy(_rays(mesh, case["rays"], seed)).cuda().double())
        return {"t": t, "prim": None, "uv": None, "nodes": None, "depth": None, "cost": None}
    if case["kind"] == "primary" and case["width"] * case["height"] * SCENES[case["scene"]][3] <= _EXACT_TESTS:
        mesh = _mesh(case["scene"])
        cam = _camera(mesh, random.Random(seed), case["width"], case["height"])
        eye, front, up = (np.array(list(v), np.float64) for v in (cam.position, cam.front, cam.up))
        f = front / np.linalg.norm(front)
        s = np.cross(f, up)
        s /= np.linalg.norm(s)
        u = np.cross(s, f)
        tan = math.tan(math.radians(float(cam.yfov_deg)) / 2)
        x = (2 * (np.arange(cam.width) + 0.5) / cam.width - 1) * tan * cam.width / cam.height
        y = (1 - 2 * (np.arange(cam.height) + 0.5) / cam.height) * tan
        d = x[None, :, None] * s + y[:, None, None] * u + f
        d /= np.linalg.norm(d, axis=2, keepdims=True)
        rays = np.zeros((cam.width * cam.height, 8))
        rays[:, 0:3], rays[:, 4:7], rays[:, 7] = eye, d.reshape(-1, 3), 100.0
        rays = torch.from_numpy(rays).cuda()
        t, found = _closest_f64(mesh, rays)
        points = torch.cat([rays[:, 0:3] + rays[:, 4:7] * t[:, None], t[:, None]], 1)
        sky = torch.cat([rays[:, 4:7], torch.full_like(t[:, None], -1.0)], 1)
        near, far = 0.01, 10000.0
        w = t * (rays[:, 4:7] @ torch.from_numpy(f).cuda())
        depth = near * (far - w) / ((far - near) * w)
        shape = (cam.height, cam.width)
        return {"depth": torch.where(found, depth, 0.0).reshape(shape),
                "points": torch.where(found[:, None], points, sky).reshape(*shape, 4), "gbuffer": None}
    return None   # paths of random decisions in 32 bits: a 64-bit renderer takes other paths
