"""Performance cases: the calls that programs built on this renderer make, over the sizes
they make them at.

A case is a dict of plain values; `prepare` turns it and a seed into what a program holds
before the call (an uploaded world, views, page-locked image buffers, a camera path, a
network), `run` is one pass through the public API, `exact` its value in 64 bits where it
has one. The scenes are the library's own presets (configurations 0 to 4 of the benchmark)
at the presets' seeds; the seed of a case picks the camera path, the per-view random
streams, the sky, the network and the edits. A world is generated and uploaded once per
process and shared by the views on it, as in a program that keeps its scene; only the
edited world belongs to one state.
"""
import ctypes
import math

import numpy as np
import torch

import smallproject_gb300 as vx

PATH_FRAMES = 240          # frames of one pass over a camera path


# ---- the cases ---------------------------------------------------------------------------

def listed():
    return [
        # A host application that owns all device memory renders a small view into its own
        # buffer (vxr_render_frame_noalloc): the smallest call, bound by latency.
        {"name": "noalloc_256x144", "kind": "noalloc", "scene": 0, "extent": 256, "emitters": 64, "model": "point",
         "w": 256, "h": 144, "cand": 32},
        # Configuration 0, an interactive viewer: one frame at a time, each waited for and
        # read back, accumulating while the camera rests.
        {"name": "still_point_640x360", "kind": "frame", "scene": 0, "extent": 256, "emitters": 64, "model": "point",
         "w": 640, "h": 360, "cand": 32, "frames": 1, "accumulate": 1, "reuse": 1},
        # A resized preview window: odd sizes, ragged tiles, area lights, 8 candidates.
        {"name": "preview_area_333x187", "kind": "frame", "scene": 0, "extent": 256, "emitters": 500, "model": "area",
         "w": 333, "h": 187, "cand": 8, "frames": 1, "accumulate": 0, "reuse": 1},
        # Configuration 1 as video: pipelined host images along a camera path.
        {"name": "video_area_1280x720", "kind": "frame", "scene": 1, "extent": 1024, "emitters": 4096, "model": "area",
         "w": 1280, "h": 720, "cand": 32, "frames": 4, "accumulate": 0, "reuse": 1},
        # Configuration 3, the benchmark's workload with the plain method: 65,536 emitters.
        {"name": "video_area_1920x1080", "kind": "frame", "scene": 3, "extent": 1024, "emitters": 65536,
         "model": "area", "w": 1920, "h": 1080, "cand": 32, "frames": 4, "accumulate": 0, "reuse": 1},
        # The benchmark's workload with the learned proposal: 4 candidates, one network
        # evaluation per pixel (the default). Evaluations shared by runs of pixels follow
        # the order of the hit list, which no two frames have alike, so their images
        # cannot be compared.
        {"name": "learned_1920x1080", "kind": "learned", "scene": 3, "extent": 1024, "emitters": 65536,
         "model": "area", "w": 1920, "h": 1080, "cand": 4, "frames": 4},
        # Loss and gradient of the proposal on a caller's samples, at the training batch
        # the benchmark uses (a program that trains offline from stored samples).
        {"name": "gradient_65536", "kind": "gradient", "batch": 65536, "clusters": 256},
        # Configuration 3 under a sky dome.
        {"name": "sky_area_1920x1080", "kind": "sky", "scene": 3, "extent": 1024, "emitters": 65536, "model": "area",
         "w": 1920, "h": 1080, "cand": 32, "frames": 2},
        # Ground truth: path-traced samples accumulated, the image read at the end.
        {"name": "truth_1920x1080", "kind": "truth", "scene": 3, "extent": 1024, "emitters": 65536, "w": 1920, "h": 1080,
         "samples": 8},
        # Configuration 2: eight views of eight worlds, mixed sizes and light models,
        # rendered as one batch per frame (a server drawing several users' views).
        {"name": "batch_8_views", "kind": "batch", "views": 8, "spec_seed": 3, "scale": 1.0, "frames": 2, "graph": 1,
         "chains": 2},
        # Configuration 4's world (1,048,576 emitters) at 4K, one waited frame: the largest.
        {"name": "still_area_3840x2160", "kind": "frame", "scene": 4, "extent": 1024, "emitters": 1048576,
         "model": "area", "w": 3840, "h": 2160, "cand": 32, "frames": 1, "accumulate": 0, "reuse": 1},
        # A game that digs and fills: some 900 voxels change, then the frame is drawn and
        # read back (the edits are committed by the frame).
        {"name": "edits_1280x720", "kind": "edits", "scene": 2, "extent": 512, "emitters": 1024, "model": "area",
         "w": 1280, "h": 720, "cand": 32, "radius": 6},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["frame", "learned", "gradient", "sky", "truth", "batch", "noalloc", "edits"],
                       [8, 3, 2, 2, 2, 2, 2, 2])[0]
    if kind == "gradient":
        return {"kind": kind, "batch": _log(rng, 1000, 131072), "clusters": rng.choice([16, 64, 128, 256])}
    if kind == "batch":
        return {"kind": kind, "views": rng.randint(2, 8), "spec_seed": rng.randint(1, 30),
                "scale": round(rng.uniform(0.3, 0.8), 3), "frames": rng.randint(1, 3), "graph": rng.randint(0, 1),
                "chains": rng.randint(1, 2)}
    w = _log(rng, 160, 256) if kind == "noalloc" else _log(rng, 300, 2048)
    h = max(64, int(w * rng.uniform(0.45, 0.8)))
    extent = rng.choice([256, 512, 1024])
    c = {"kind": kind, "scene": 3 if kind == "learned" else rng.choice([0, 1, 2, 3]), "extent": extent,
         "emitters": _log(rng, 2048 if kind == "learned" else 16, 65536), "model": rng.choice(["area", "area", "point"]),
         "w": w, "h": h, "cand": rng.choice([4, 8, 16, 32, 32])}
    most = max(1, 8000000 // (w * h))      # frames: no pass draws more pixels than the 4K frame
    if kind == "frame":
        c.update(frames=min(most, rng.randint(1, 4)), accumulate=rng.randint(0, 1), reuse=rng.choice([1, 1, 1, 0]))
    elif kind == "learned":
        c.update(model="area", cand=rng.choice([1, 2, 4, 8, 12]), frames=min(most, rng.randint(1, 4)))
    elif kind == "sky":
        c.update(frames=rng.randint(1, 2))
    elif kind == "truth":
        c.update(samples=rng.randint(1, 8))
        del c["model"], c["cand"]
    elif kind == "edits":
        c.update(extent=rng.choice([256, 512]), scene=rng.choice([0, 2]), radius=rng.randint(2, 9))
        c["emitters"] = min(c["emitters"], 4096)
    return c


# ---- what a program holds ------------------------------------------------------------------

def _images(pixels, n):
    """n page-locked float4 images."""
    return [torch.empty(pixels, 4, dtype=torch.float32, pin_memory=True) for _ in range(n)]


_worlds = {}


def _preset(case):
    return vx.scene_preset(case["scene"], extent=case["extent"], emitters=case["emitters"])


def _world(case, clusters=0):
    """The uploaded world of a case's scene, made once per process."""
    key = (case["scene"], case["extent"], case["emitters"], clusters)
    if key not in _worlds:
        if len(_worlds) > 24:
            _worlds.clear()
        w = vx.World()
        w.generate(_preset(case))
        if clusters:
            w.cluster_lights(clusters, 1, 8)
        w.upload()
        _worlds[key] = w
    return _worlds[key]


def _model(case):
    return vx.LIGHTS_POINT if case["model"] == "point" else vx.LIGHTS_AREA


def _view(world, case, seed, **kw):
    return vx.View(world, vx.view_desc(case["w"], case["h"], _model(case), num_candidates=case["cand"],
                                       rng_seed=(seed * 2654435761 + 12345) & 0xFFFFFFFF or 1, **kw))


def _path(desc, seed):
    """Pose of frame f on a seeded camera path."""
    return lambda f: vx.camera_path(desc, 1 + seed % 100003, f % PATH_FRAMES, PATH_FRAMES)


def _still(desc, seed):
    """A resting camera: one pose of the path."""
    pose = vx.camera_path(desc, 1 + seed % 100003, seed % PATH_FRAMES, PATH_FRAMES)
    return lambda f: pose


def _sky(seed):
    """A clear sky with a sun (float32[512, 1024, 4]) and blue-noise tables of hashed bytes."""
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:512, 0:1024].astype(np.float32)
    up = np.clip(1.0 - y / 256.0, 0.0, 1.0)[..., None]
    tex = np.concatenate([0.3 + 0.4 * up, 0.4 + 0.5 * up, 0.6 + 0.9 * up, np.ones_like(up)], axis=2).astype(np.float32)
    sx, sy = rng.integers(100, 924), rng.integers(40, 200)
    tex[..., :3] += (40.0 * np.exp(-((x - sx) ** 2 + (y - sy) ** 2) / 60.0))[..., None].astype(np.float32)
    return tex, rng.integers(0, 256, vx.BLUE_NOISE_WORDS, dtype=np.uint32)


def _network(view, seed):
    """A network away from its initial one: encodings of the size training gives them and a
    peaked output layer, so the softmax favours some clusters as a trained one does."""
    p = view.proposal_params()
    K = view.proposal_shape()[1]
    tables = 2 * (1 << 16) * 8
    p[:tables] *= 4000.0
    out = len(p) - K - K * 64
    p[out:out + K * 64] *= 1.5
    rng = np.random.default_rng(seed)
    p[out + K * 64:] = rng.normal(0.0, 0.5, K).astype(np.float32)
    view.proposal_set_params(p)
    return p


def _samples(case, seed):
    """Shading points of a terrain, target clusters and heavy-tailed weights, as stored by a
    program that trains from its reservoirs."""
    rng = np.random.default_rng(seed)
    B = case["batch"]
    s = np.zeros((B, 4), np.float32)
    s[:, 0] = rng.uniform(0.0, 1024.0, B)
    s[:, 2] = rng.uniform(0.0, 1024.0, B)
    s[:, 1] = 300.0 + 90.0 * np.sin(s[:, 0] / 97.0) + 70.0 * np.cos(s[:, 2] / 61.0) + rng.uniform(-8.0, 8.0, B)
    s[:, 3] = rng.choice(6, B, p=[0.1, 0.5, 0.1, 0.1, 0.1, 0.1]).astype(np.uint32).view(np.float32)
    near = (s[:, 0] / 128.0).astype(np.int64) * 8 + (s[:, 2] / 128.0).astype(np.int64)
    target = ((near * 37 + rng.integers(0, 7, B)) % case["clusters"]).astype(np.uint32)
    weight = np.exp(rng.normal(0.0, 1.0, B)).astype(np.float32)
    weight[rng.random(B) < 0.1] = 0.0
    return s, target, weight


def prepare(case, seed):
    seed = int(seed)
    kind = case["kind"]
    s = {"case": case, "f": 0}
    if kind == "gradient":
        scene = {"scene": 1, "extent": 1024, "emitters": 4096}
        world = _world(scene, case["clusters"])
        view = vx.View(world, vx.view_desc(64, 64, vx.LIGHTS_AREA))
        view.proposal_enable(seed=1 + seed % 1000003, batch=case["batch"])
        s.update(view=view, params=_network(view, seed))
        s["samples"], s["target"], s["weight"] = _samples(case, seed)
        return s
    if kind == "batch":
        worlds, views, paths, images = [], [], [], []
        from smallproject_gb300 import workloads
        for i, sp in enumerate(workloads.config2_specs(case["spec_seed"], case["views"], case["scale"])):
            c = {"scene": 1, "extent": sp["extent"], "emitters": sp["emitters"], "model": sp["light_model"],
                 "w": sp["width"], "h": sp["height"], "cand": 32}
            worlds.append(_world(c))
            views.append(_view(worlds[-1], c, seed * 16 + i))
            paths.append(_path(_preset(c), seed * 16 + i))
            images.append(_images(views[-1].n, 1)[0])
        batch = vx.Batch(views, graph=bool(case["graph"]), chains=min(case["chains"], len(views)))
        s.update(batch=batch, views=views, paths=paths, images=images)
        return s
    desc = _preset(case)
    if kind == "noalloc":
        world = _world(case)
        grid, bricks, lights = world.arrays()
        cam = vx.Camera((seed * 7919 + 1) & 0xFFFFFFFF)
        dev = lambda a: torch.from_numpy(a.view(np.int32).reshape(-1).copy()).cuda()  # noqa: E731
        s.update(cam=cam, path=_path(desc, seed), grid=dev(grid), bricks=dev(bricks),
                 lights=dev(np.ascontiguousarray(lights).view(np.uint32)), nbricks=len(bricks), nlights=len(lights),
                 out=torch.zeros(case["h"], case["w"], 4, dtype=torch.float32, device="cuda"))
        return s
    if kind == "truth":
        world = _world(case)
        view = vx.View(world, vx.view_desc(case["w"], case["h"], vx.LIGHTS_AREA, accumulate=1,
                                           rng_seed=(seed * 2654435761 + 12345) & 0xFFFFFFFF or 1))
        s.update(view=view, path=_still(desc, seed), images=_images(view.n, 1))
        return s
    if kind == "edits":
        world = vx.World()
        world.generate(desc)
        rng = np.random.default_rng(seed)
        r = case["radius"]
        g = np.arange(-r, r + 1)
        x, y, z = np.meshgrid(g, g, g, indexing="ij")
        ball = (x * x + y * y + z * z <= r * r).reshape(-1)
        s["ball"] = ((x + r) | ((y + r) << 10) | ((z + r) << 20)).reshape(-1)[ball].astype(np.uint32)
        at = rng.integers(2 * r + 2, desc.extent - 2 * r - 2, (64, 2))
        s["holes"] = [(int(a), max(int(vx.scene_height(desc, int(a), int(b))), r + 1), int(b)) for a, b in at]
        s["rock"] = (np.uint32(0xF000) | rng.integers(0x111, 0xFFF, len(s["ball"]), dtype=np.uint32)).astype(np.uint32)
        s["air"] = np.zeros(len(s["ball"]), np.uint32)
        view = _view(world, case, seed)
        s.update(world=world, view=view, path=_path(desc, seed), images=_images(view.n, 1))
        return s
    if kind == "learned":
        world = _world(case, 256)
        view = _view(world, case, seed)
        view.proposal_enable(seed=1 + seed % 1000003)
        _network(view, seed)
        view.proposal_use(True)
    else:
        world = _world(case)
        kw = {}
        if kind == "frame":
            kw = {"accumulate": case["accumulate"], "spatial": case["reuse"], "temporal": case["reuse"]}
        view = _view(world, case, seed, **kw)
    if kind == "sky":
        tex, noise = _sky(seed)
        view.set_sky(tex, None, 0.5, noise)
    still = kind == "frame" and case["accumulate"]
    s.update(view=view, path=(_still if still else _path)(desc, seed), images=_images(view.n, case["frames"]))
    return s


# ---- one pass --------------------------------------------------------------------------------

def _read_accum(view, out):
    vx.check(vx.load().vxr_view_read_accum(view.h, ctypes.cast(out.data_ptr(), ctypes.POINTER(ctypes.c_float))))


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "gradient":
        return list(s["view"].proposal_grad(s["samples"], s["target"], s["weight"]))
    if kind == "noalloc":
        s["cam"].lookat(*s["path"](s["f"]))
        k = s["cam"].begin_frame(case["w"], case["h"])
        k.accumulate, k.spatial, k.temporal = 0, 1, 0
        k.numberOfLights, k.numberOfCandidates = s["nlights"], case["cand"]
        k.numberOfMaxTemporalImportance, k.spatialRadius, k.spatialTaps = 20, 30, 5
        vx.check(vx.load().vxr_render_frame_noalloc(
            s["grid"].data_ptr(), s["bricks"].data_ptr(), s["nbricks"], s["lights"].data_ptr(), s["nlights"],
            _model(case), ctypes.byref(k), s["out"].data_ptr(), torch.cuda.current_stream().cuda_stream))
        s["cam"].end_frame()
        s["f"] += 1
        return s["out"]
    if kind == "batch":
        for _ in range(case["frames"]):
            for v, path in zip(s["views"], s["paths"]):
                v.lookat(*path(s["f"]))
            s["batch"].render()
            s["f"] += 1
        s["batch"].wait()
        for v, im in zip(s["views"], s["images"]):
            _read_accum(v, im)
        return list(s["images"])
    view, images = s["view"], s["images"]
    if kind == "truth":
        view.lookat(*s["path"](s["f"]))
        for _ in range(case["samples"]):
            view.begin_frame()
            view.stage(vx.STAGE_PATH_TRACE)
            view.stage(vx.STAGE_ACCUMULATE)
            view.end_frame()
        s["f"] += 1
        _read_accum(view, images[0])
        return images[0]
    if kind == "edits":
        x, y, z = s["holes"][s["f"] % len(s["holes"])]
        r = case["radius"]
        fill = (s["f"] // len(s["holes"]) + s["f"]) % 2
        s["world"].stamp(s["ball"], s["rock"] if fill else s["air"], (x - r, y - r, z - r))
    frames = case.get("frames", 1)
    if frames == 1:
        view.render_to_host(*s["path"](s["f"]), images[0].numpy())
        s["f"] += 1
        return images[0]
    last = None
    for i in range(frames):
        ticket = view.render_to_host_async(*s["path"](s["f"]), images[i].numpy())
        s["f"] += 1
        if last is not None:
            view.image_wait(last)
        last = ticket
    view.image_wait(last)
    return list(images)


# ---- what a pass cannot do without -------------------------------------------------------------

def _frame_work(w, h, cand, model, emitters, extent, reuse=1):
    """Bytes and operations of one frame: per pixel the image out (16), the accumulator
    (16), G-buffer out and previous one in (16), reservoir out and history in (64); the
    light table and the map's cells once. Operations: a primary ray (some 100 cells of 8),
    two shadow rays (some 50 cells each), the candidates, five spatial taps."""
    px = w * h
    c = min(cand, emitters)
    nbytes = px * (16 + 16 + (80 if reuse else 0)) + emitters * 32 + (extent // 8) ** 3 * 4
    flops = px * (800 + 2 * 400 + c * (160 if model == "area" else 50) + (5 * 60 if reuse else 0))
    return nbytes, flops


def work(case):
    kind = case["kind"]
    if kind == "gradient":
        B, K = case["batch"], case["clusters"]
        mlp = 64 * 32 + 2 * 64 * 64 + 64 * K
        n = 2 * (1 << 16) * 8 + mlp + 3 * 64 + K
        return {"bytes": float(B * 24 + 2 * n * 4), "flops": float(6 * B * mlp + 4 * B * 2 * 8 * 8)}
    if kind == "batch":
        from smallproject_gb300 import workloads
        b = f = 0
        for sp in workloads.config2_specs(case["spec_seed"], case["views"], case["scale"]):
            x, y = _frame_work(sp["width"], sp["height"], 32, sp["light_model"], sp["emitters"], sp["extent"])
            b += x
            f += y
        return {"bytes": float(b * case["frames"]), "flops": float(f * case["frames"])}
    if kind == "truth":
        px = case["w"] * case["h"]
        return {"bytes": float(px * 32 * case["samples"] + (case["extent"] // 8) ** 3 * 4),
                "flops": float(px * 1250 * case["samples"])}
    b, f = _frame_work(case["w"], case["h"], case["cand"], case["model"], case["emitters"], case["extent"],
                       0 if kind == "noalloc" else case.get("reuse", 1))
    n = case.get("frames", 1)
    if kind == "learned":
        mlp = 64 * 32 + 2 * 64 * 64 + 64 * 256
        f += case["w"] * case["h"] * 2 * mlp
    if kind == "sky":
        f += case["w"] * case["h"] * 200
        b += 1024 * 512 * 16
    return {"bytes": float(b * n), "flops": float(f * n)}


# ---- 64-bit values -------------------------------------------------------------------------------

def exact(case, seed):
    """Loss and gradient of the proposal in 64 bits. Images have no such value: which emitter
    a pixel's reservoir holds, and whether a ray is stopped, are choices that 64-bit
    arithmetic makes otherwise, so an image computed that way is another sample."""
    if case["kind"] != "gradient":
        return None
    B, K, T, H = case["batch"], case["clusters"], 1 << 16, 64
    samples, target, weight = _samples(case, int(seed))
    p = torch.from_numpy(np.array(prepare(case, seed)["params"])).cuda().double()
    sizes = [("enc", (2 * T, 8)), ("W1", (H, 32)), ("b1", (H,)), ("W2", (H, H)), ("b2", (H,)), ("W3", (H, H)),
             ("b3", (H,)), ("W4", (K, H)), ("b4", (K,))]
    P, o = {}, 0
    for name, shape in sizes:
        n = int(np.prod(shape))
        P[name] = p[o:o + n].reshape(shape).clone().requires_grad_(True)
        o += n
    pos = torch.from_numpy(samples[:, :3].copy()).cuda()
    code = torch.from_numpy(samples[:, 3].copy().view(np.int32).astype(np.int64)).cuda()
    cols = []
    for level, R in enumerate((32, 128)):
        u = (pos * (R / 1024.0)).clamp(0.0, float(R))
        i = u.long().clamp(max=R - 1)
        f = (u - i).double()
        x = torch.zeros(B, 8, dtype=torch.float64, device="cuda")
        for q in range(8):
            on = torch.tensor([q & 1, (q >> 1) & 1, q >> 2], device="cuda")
            c = i + on
            h = c[:, 0] ^ ((c[:, 1] * 2654435761) & 0xFFFFFFFF) ^ ((c[:, 2] * 805459861) & 0xFFFFFFFF)
            wq = torch.where(on == 1, f, 1.0 - f).prod(1)
            x = x + wq[:, None] * P["enc"][level * T + (h & (T - 1))]
        cols.append(x)
    onehot = torch.nn.functional.one_hot(code, 16).double()
    X = torch.cat(cols + [onehot], dim=1)
    h = torch.relu(X @ P["W1"].T + P["b1"])
    h = torch.relu(h @ P["W2"].T + P["b2"])
    h = torch.relu(h @ P["W3"].T + P["b3"])
    logp = torch.log_softmax(h @ P["W4"].T + P["b4"], dim=1)
    w = torch.from_numpy(weight).cuda().double()
    t = torch.from_numpy(target.astype(np.int64)).cuda()
    loss = -(w / w.sum() * logp[torch.arange(B, device="cuda"), t]).sum()
    grads = torch.autograd.grad(loss, [P[n] for n, _ in sizes])
    return [float(loss), torch.cat([g.reshape(-1) for g in grads])]
