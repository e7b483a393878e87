"""What the renderer is measured on: the work its users have it do.

Each case is one of the framework's calls at a size that its benchmark
workloads, tests or serving defaults use, through the public entry points of
the Python package.  The scene set of a rendering case is the handle that a
program keeps (the same for every seed, built once); the camera poses, depth
images, colours and noise seeds are the inputs and follow the seed.

Kinds of cases:
  draw       update the cameras from host arrays, draw, optionally ambient
             occlusion; the output planes of the framebuffer
  serve      one continuous-batching step of the request server, images in
             pinned host memory
  replay     one camera keyframe per environment, rendered into CUDA tensors
  noise      depth-sensor noise on one image or on a batch of images
  occlusion  ambient occlusion on one caller-owned image
  unproject  window depth to metres on a caller-owned image
"""
import functools
import math

import numpy as np
import torch

import __graft_entry__

pkg = __graft_entry__.load_package()

from habitat_sim_gb300 import noise, procedural, server  # noqa: E402


# ------------------------------------------------------------------- cases
def listed():
    return [
        # One agent asks for one frame of its room (interactive use, evaluation
        # of a single episode): the plain draw call, where latency counts.
        dict(name="one view", kind="draw", scene="rooms", scenes=1, envs=1, width=128, height=128,
             mode="plain"),
        # 16 agents in one room: the smallest vectorised environment of the
        # benchmark, batched.
        dict(name="16 views of a room", kind="draw", scene="rooms", scenes=1, envs=16, width=128,
             height=128, mode="batched"),
        # The headline workload: 1024 agents over 4 furnished, textured rooms.
        dict(name="1024 textured views", kind="draw", scene="furnished", scenes=4, envs=1024, width=128,
             height=128, mode="batched"),
        # The plain per-scene draw, the library's default mode, on a batch of
        # furnished rooms with an unusual image size.
        dict(name="48 plain views", kind="draw", scene="furnished", scenes=4, envs=48, width=160,
             height=120, mode="plain"),
        # Mixed curriculum: scenes of very different size, resolutions of 64,
        # 128 and 256, individual fields of view, ragged framebuffer.
        dict(name="512 mixed views", kind="draw", scene="mixed", scenes=12, envs=512, width=0, height=0,
             mode="batched"),
        # Scanned buildings: dense sub-pixel triangles with vertex colours.
        dict(name="64 views of scans", kind="draw", scene="scans", scenes=2, envs=64, width=256,
             height=256, mode="batched"),
        # Lit rooms: Phong materials, three lights, trilinear mipmapped
        # textures, then ambient occlusion on every frame.
        dict(name="128 lit views with AO", kind="draw", scene="lit", scenes=2, envs=128, width=128,
             height=128, mode="batched", occlusion="classic"),
        # A full step of the request server's default slots (96 + 160 + 64
        # requests of 64, 128 and 256 px), scenes resident.
        dict(name="serve 320 requests", kind="serve", scenes=24, s64=96, s128=160, s256=64),
        # Re-rendering recorded episodes: a keyframe per environment.
        dict(name="replay 256 episodes", kind="replay", scenes=4, envs=256, width=128, height=128),
        # Sensor noise on the depth of every environment of a batch.
        dict(name="noise on 1024 images", kind="noise", images=1024, width=128, height=128, layout="tiles"),
        # Ambient occlusion on one camera image of a robot.
        dict(name="AO on one 640x480 image", kind="occlusion", width=640, height=480,
             algorithm="classic", blur="bilateral"),
        # Metres from the window-depth plane of a large framebuffer.
        dict(name="unproject 4096x4096", kind="unproject", width=4096, height=4096, padding=0),
    ]


def _log(rng, lo, hi):
    """An integer in [lo, hi], its logarithm uniform."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rooms", "furnished", "mixed", "scans", "lit", "serve", "replay", "noise", "noise",
                       "occlusion", "occlusion", "unproject"])
    if kind in ("rooms", "furnished", "lit"):
        mode = rng.choice(["plain", "batched", "batched"])
        envs = _log(rng, 1, 64 if mode == "plain" else 384)
        w = _log(rng, 33, 320)
        c = dict(kind="draw", scene=kind, scenes=1 if envs < 8 else rng.randint(1, 4), envs=envs, width=w,
                 height=max(16, int(w * rng.uniform(0.5, 1.2))), mode=mode)
        if envs * c["width"] * c["height"] > 1 << 23:
            c["envs"] = max(1, (1 << 23) // (c["width"] * c["height"]))
        if kind == "lit" and rng.random() < 0.5:
            c["occlusion"] = rng.choice(["classic", "cache_aware"])
        return c
    if kind == "mixed":
        return dict(kind="draw", scene="mixed", scenes=rng.randint(2, 12), envs=_log(rng, 8, 400), width=0,
                    height=0, mode="batched")
    if kind == "scans":
        w = _log(rng, 96, 280)
        return dict(kind="draw", scene="scans", scenes=rng.randint(1, 2), envs=_log(rng, 1, 48), width=w,
                    height=w, mode="batched")
    if kind == "serve":
        return dict(kind="serve", scenes=rng.randint(4, 24), s64=_log(rng, 1, 96), s128=_log(rng, 1, 160),
                    s256=_log(rng, 1, 64))
    if kind == "replay":
        return dict(kind="replay", scenes=rng.randint(1, 4), envs=_log(rng, 2, 250),
                    width=_log(rng, 48, 160), height=_log(rng, 48, 160))
    if kind == "noise":
        if rng.random() < 0.4:
            return dict(kind="noise", images=1, width=_log(rng, 61, 1920), height=_log(rng, 47, 1080),
                        layout="one")
        return dict(kind="noise", images=_log(rng, 2, 900), width=_log(rng, 33, 140),
                    height=_log(rng, 33, 130), layout=rng.choice(["tiles", "ragged"]))
    if kind == "occlusion":
        return dict(kind="occlusion", width=_log(rng, 61, 1920), height=_log(rng, 47, 1080),
                    algorithm=rng.choice(["classic", "cache_aware"]),
                    blur=rng.choice(["bilateral", "bilateral", "special", "none"]))
    return dict(kind="unproject", width=_log(rng, 61, 4000), height=_log(rng, 47, 4000),
                padding=rng.choice([0, 0, 1, 12]))


# ------------------------------------------------------------------ scenes
@functools.lru_cache(maxsize=3)
def _workload(scene, scenes, envs, width, height):
    """The scene set of a rendering case and its environments."""
    if scene == "rooms":
        wl = procedural.config0(seed=21, envs=envs)
    elif scene == "scans":
        wl = procedural.config3(seed=22, envs=envs, scenes=scenes, edge=0.026)
    elif scene == "mixed":
        wl = procedural.config2(seed=23, envs=envs, scenes=scenes, tri_range=(2e4, 5e5), texture_size=256)
    elif scene == "lit":
        wl = procedural.config1(seed=24, envs=envs, scenes=scenes, instances=60, texture_size=256)
    else:
        wl = procedural.config1(seed=25, envs=envs, scenes=scenes)
    if wl.uniform:
        wl.viewports = [(width, height)] * envs
    return wl


@functools.lru_cache(maxsize=2)
def _catalog(scenes):
    return server.SceneCatalog(scenes, seed=26, tri_range=(1e4, 3e5), texture_side=512,
                               pool_bytes=64 << 20)


def _normals(mesh):
    """Vertex normals: the mean of the normals of the triangles around each."""
    p, t = mesh["positions"].astype(np.float64), mesh["indices"].reshape(-1, 3)
    n = np.cross(p[t[:, 1]] - p[t[:, 0]], p[t[:, 2]] - p[t[:, 0]])
    out = np.zeros_like(p)
    for k in range(3):
        np.add.at(out, t[:, k], n)
    length = np.linalg.norm(out, axis=1, keepdims=True)
    return (out / np.where(length > 0, length, 1.0)).astype(np.float32)


def _lit_renderer(wl, mode, planes):
    """The workload with Phong materials, mipmapped textures and three lights."""
    cfg = pkg.RendererConfiguration().setTileSizeCount(wl.viewports[0], procedural.grid_for(wl.envs))
    cfg.setDrawMode(mode).setPlanes(planes).setMaxLightCount(3)
    r = pkg.RendererStandalone(cfg, pkg.RendererStandaloneConfiguration().setFlags(
        pkg.RendererStandaloneFlags.QuietLog))
    tex = [r.addTexture(t["pixels"], 1, 0, 0, minFilter=2, mipFilter=2, generateMipmap=True)
           for t in wl.textures]
    mesh = [r.addMesh(m["positions"], m["colors"], m["texcoords"], m["object_ids"], m["indices"],
                      normals=_normals(m)) for m in wl.meshes]
    mats = [r.addMaterial(c, 0 if t < 0 else tex[t], layer, shaded=True) for (c, t, layer) in wl.materials]
    for name, views in wl.templates:
        r.addNodeHierarchyTemplate(name, [(mesh[m], o, n, mats[k], None) for (m, o, n, k) in views])
    for e in range(wl.envs):
        for (template, bake, sid) in wl.instances[wl.scene_of_env[e]]:
            r.setSemanticId(e, r.addNodeHierarchy(e, template, bake), sid)
        nodes = [r.addEmptyNode(e) for _ in range(3)]
        for node, kind in zip(nodes, (pkg.RendererLightType.Point, pkg.RendererLightType.Point,
                                      pkg.RendererLightType.Directional)):
            r.addLight(e, node, kind)
        move = r.transformations(e)
        move[nodes[0], 3, :3] = (-2.0, 2.6, 1.0)
        move[nodes[1], 3, :3] = (2.5, 2.2, -1.5)
        move[nodes[2], 2, :3] = (0.3, 0.9, 0.3)
        r.lightColors(e)[:] = ((3.0, 2.8, 2.5), (2.0, 2.2, 2.6), (0.3, 0.3, 0.3))
        r.lightRanges(e)[:2] = 12.0
    return r


def _poses(wl, seed):
    """A camera per environment: anywhere in the room, slightly tilted."""
    rng = np.random.default_rng([seed, 31])
    n, rx, rz = wl.envs, wl.room[0] / 2 - 0.3, wl.room[2] / 2 - 0.3
    views = server.pose_views(rng.uniform(-rx, rx, n), rng.uniform(1.0, 1.6, n), rng.uniform(-rz, rz, n),
                              rng.uniform(0, 2 * math.pi, n), np.radians(rng.uniform(-15, 15, n)),
                              np.zeros(n))
    projections = np.stack([procedural.projection(wl.hfov[e], *wl.viewports[e]) for e in range(n)])
    return projections.astype(np.float32), views


def _room_depth(width, height, seed, images=1):
    """Metres along the view axis seen by cameras in boxy rooms with spheres
    (hfov 90, 0 where the far plane is reached), [images, height, width]."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def u(lo, hi, *shape):
        return torch.rand(images, *shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo

    out = torch.empty(images, height, width, device="cuda", dtype=torch.float32)
    yaw, eye = u(0, 2 * math.pi), u(-1.0, 1.0, 3)
    half, far = u(1.5, 6.5, 3), 10.0
    centre, radius = u(-2.5, 2.5, 12, 3), u(0.15, 0.8, 12)
    x = (torch.arange(width, device="cuda", dtype=torch.float64) * 2 + 1 - width) / width
    y = (torch.arange(height, device="cuda", dtype=torch.float64) * 2 + 1 - height) / width
    for i in range(images):
        c, s = torch.cos(yaw[i]), torch.sin(yaw[i])
        d = torch.stack([(c * x + s).expand(height, width), y[:, None].expand(height, width),
                         (c - s * x).expand(height, width)], -1)
        t = torch.where(d == 0, math.inf, (half[i] * torch.sign(d) - eye[i] * 0.5) / d).amin(-1)
        o = eye[i] * 0.5 - centre[i]
        a, b = (d * d).sum(-1, keepdim=True), d @ o.T
        disc = b * b - a * ((o * o).sum(-1) - radius[i] ** 2)
        near = (-b - disc.clamp(min=0).sqrt()) / a
        near = torch.where((disc > 0) & (near > 0.05), near, math.inf).amin(-1)
        t = torch.minimum(t, near)
        out[i] = torch.where(t < far, t, 0.0)
    return out


# ----------------------------------------------------------------- prepare
_one_stream = []


def _stream():
    """The stream on which a program's draws follow one another."""
    if not _one_stream:
        _one_stream.append(torch.cuda.Stream())
    return _one_stream[0]


def _draw_planes(case):
    # The benchmark's planes: colour, metres, ids; a single agent takes all.
    if case["envs"] == 1:
        return pkg.Plane.All
    return pkg.Plane.Color | pkg.Plane.LinearDepth | pkg.Plane.Semantic


def prepare(case, seed):
    return dict({"draw": _prepare_draw, "serve": _prepare_serve, "replay": _prepare_replay,
                 "noise": _prepare_noise, "occlusion": _prepare_occlusion,
                 "unproject": _prepare_unproject}[case["kind"]](case, seed), kind=case["kind"])


def run(state):
    return {"draw": _run_draw, "serve": _run_serve, "replay": _run_replay, "noise": _run_noise,
            "occlusion": _run_occlusion, "unproject": _run_unproject}[state["kind"]](state)


def _case_workload(case):
    return _workload(case["scene"], case["scenes"], case["envs"], case["width"], case["height"])


def _prepare_draw(case, seed):
    wl = _case_workload(case)
    mode = pkg.DrawMode.PerScene if case["mode"] == "plain" else pkg.DrawMode.Batched
    planes = _draw_planes(case)
    r = (_lit_renderer(wl, mode, planes) if case["scene"] == "lit" else
         procedural.build_renderer(pkg, wl, mode=mode, planes=planes))
    occlusion = None
    if case.get("occlusion"):
        occlusion = pkg.HbaoConfiguration()
        if case["occlusion"] == "cache_aware":
            occlusion.setAlgorithm(pkg.HbaoType.CacheAware)
    out = {"color": r.colorTensor(), "linear": r.linearDepthTensor(),
           "semantic": r.semanticTensor().view(torch.int32)}
    if planes & pkg.Plane.Depth:
        out["depth"] = r.depthTensor()
    projections, views = _poses(wl, seed)
    return dict(renderer=r, projections=projections, views=views, graph=mode == pkg.DrawMode.Batched,
                occlusion=occlusion, out=out, stream=_stream())


def _run_draw(s):
    r = s["renderer"]
    r.updateCameras(s["projections"], s["views"])
    if s["graph"]:
        r.draw(s["stream"], graph=True)
    else:
        r.draw(s["stream"])
    if s["occlusion"] is not None:
        r.drawHbao(s["occlusion"], s["stream"])
    return s["out"]


def _slots(case):
    return {64: case["s64"], 128: case["s128"], 256: case["s256"]}


def _prepare_serve(case, seed):
    cat = _catalog(case["scenes"])
    srv = server.RenderServer(pkg, cat, slots=_slots(case), max_resident=len(cat),
                              max_loads_per_step=len(cat))
    warm = server.random_requests(cat, len(cat), rate=0, seed=5)
    for scene, request in enumerate(warm):  # every scene resident
        request.scene = scene
    srv.serve(warm, realtime=False, keep_images=False)
    batch = {}
    for k, (side, count) in enumerate(_slots(case).items()):
        batch[side] = server.random_requests(cat, count, rate=0, seed=3 * seed + k, classes=(side,), p=(1.0,))
    return dict(server=srv, batch=batch)


def _run_serve(s):
    handle, _ = s["server"].launch(s["batch"])
    s["server"].finish(handle, keep_images=False)
    return {"color": handle[1][0], "linear": handle[1][1], "semantic": handle[1][2].view(torch.int32)}


def _prepare_replay(case, seed):
    wl = _workload("furnished", case["scenes"], case["envs"], case["width"], case["height"])
    cfg = pkg.ReplayRendererConfiguration()
    cfg.num_environments = wl.envs
    w, h = wl.viewports[0]
    cfg.sensor_specifications = [pkg.CameraSensorSpec(resolution=(h, w), hfov=float(wl.hfov[0]),
                                                      near=procedural.NEAR, far=procedural.FAR)]
    cfg.quiet = True
    rr = pkg.ReplayRenderer.create_batch_replay_renderer(cfg)
    procedural.add_resources(rr.renderer, wl)
    loads = [procedural.scene_keyframe(pkg, wl, k).to_string() for k in range(len(wl.instances))]
    rr.set_environment_keyframes_batch([loads[wl.scene_of_env[e]] for e in range(wl.envs)])
    _, views = _poses(wl, seed)
    return dict(replay=rr, keyframes=[procedural.camera_keyframe(pkg, v).to_string() for v in views],
                color=torch.zeros(wl.envs, h, w, 4, dtype=torch.uint8, device="cuda"),
                depth=torch.zeros(wl.envs, h, w, dtype=torch.float32, device="cuda"))


def _run_replay(s):
    s["replay"].set_environment_keyframes_batch(s["keyframes"], sensor_prefix="sensor_")
    s["replay"].render(s["color"], s["depth"])
    return {"color": s["color"], "depth": s["depth"]}


def _noise_layout(case):
    """(offset, pitch, width, height) of every image of a ragged batch: widths
    and heights from a third of the case's to the whole."""
    rng = np.random.default_rng(case["images"])
    w = rng.integers(max(2, case["width"] // 3), case["width"] + 1, case["images"])
    h = rng.integers(max(2, case["height"] // 3), case["height"] + 1, case["images"])
    offset = np.concatenate([[0], np.cumsum(w * h)])[:-1]
    return np.stack([offset, w, w, h], 1).astype(np.int64)


def _noise_input(case, seed):
    n, w, h = case["images"], case["width"], case["height"]
    base = min(n, 24)  # that many rooms, again at other distances for the rest
    rooms = _room_depth(w, h, seed, base)
    scale = torch.linspace(0.7, 1.4, -(-n // base), device="cuda")
    depth = (rooms[None] * scale[:, None, None, None]).reshape(-1, h, w)[:n]
    if case["layout"] == "one":
        return depth[0].contiguous()
    if case["layout"] == "tiles":
        tx, ty = procedural.grid_for(n)
        plane = torch.zeros(ty * tx, h, w, device="cuda")
        plane[:n] = depth
        return plane.reshape(ty, tx, h, w).permute(0, 2, 1, 3).reshape(ty * h, tx * w).contiguous()
    layout = _noise_layout(case)
    return torch.cat([depth[i, :a[3], :a[2]].reshape(-1) for i, a in enumerate(layout)])


def _prepare_noise(case, seed):
    s = dict(depth=_noise_input(case, seed), case=dict(case))
    if case["layout"] == "one":
        s["model"] = noise.RedwoodDepthNoiseModel(1.0, seed=seed)
    else:
        s["model"] = noise.RedwoodNoiseModelGPUImpl(noise.load_model(), 0, 1.0, seed=seed)
        s["out"] = torch.zeros_like(s["depth"])
        s["layout"] = _noise_layout(case) if case["layout"] == "ragged" else None
        s["tiles"] = procedural.grid_for(case["images"])[0]
    return s


def _run_noise(s):
    case, depth = s["case"], s["depth"]
    if case["layout"] == "one":
        return s["model"].simulate(depth)
    if case["layout"] == "tiles":
        s["model"].simulate_tiles(depth.data_ptr(), s["out"].data_ptr(), depth.shape[1], case["width"],
                                  case["height"], s["tiles"], case["images"])
    else:
        s["model"].simulate_images(depth.data_ptr(), s["out"].data_ptr(), s["layout"])
    return s["out"]


def _prepare_occlusion(case, seed):
    w, h = case["width"], case["height"]
    cfg = pkg.HbaoConfiguration()
    if case["algorithm"] == "cache_aware":
        cfg.setAlgorithm(pkg.HbaoType.CacheAware)
    if case["blur"] == "special":
        cfg.setUseSpecialBlur(True)
    elif case["blur"] == "none":
        cfg.setNoBlur(True)
    g = torch.Generator(device="cuda").manual_seed(seed)
    color = torch.randint(40, 256, (h, w, 4), generator=g, device="cuda", dtype=torch.uint8)
    return dict(config=cfg, projection=procedural.projection(90.0, w, h), color=color,
                depth=_room_depth(w, h, seed)[0].contiguous())


def _run_occlusion(s):
    color = s["color"].clone()  # the camera's own image stays as it was
    pkg.hbaoApply(s["config"], s["projection"], s["depth"], color)
    return color


def _unprojection():
    return pkg.calculateDepthUnprojection(procedural.projection(90.0, 128, 128))


def _unproject_input(case, seed):
    h, w = case["height"], case["width"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    metres = torch.rand(h, w, generator=g, device="cuda") * 9.0 + 0.2
    a, b = (float(v) for v in _unprojection())
    window = torch.empty(h, w + case["padding"], device="cuda")
    window[:, :w] = b / metres - a
    window[:, w:] = 0.5
    window[: h // 8, :w] = 1.0  # background
    return window


def _prepare_unproject(case, seed):
    return dict(window=_unproject_input(case, seed), unprojection=_unprojection(), width=case["width"])


def _run_unproject(s):
    depth = s["window"].clone()  # the window-depth plane stays as it was
    pkg.unprojectDepthDevice(s["unprojection"], depth[:, :s["width"]])
    return depth


# -------------------------------------------------------------------- work
def work(case):
    """Bytes that one pass cannot do without (inputs once, outputs once); the
    geometry and textures of the scenes count as inputs of a draw."""
    k = case["kind"]
    if k == "draw":
        wl = _case_workload(case)
        px = sum(w * h for (w, h) in wl.viewports)
        planes = 16 if case["envs"] == 1 else 12
        flops = 60 * float(px) + (32 * 40 * float(px) if case.get("occlusion") else 0.0)
        return {"bytes": float(px * planes + wl.geometry_bytes()), "flops": flops}
    if k == "serve":
        cat = _catalog(case["scenes"])
        px = sum(side * side * n for side, n in _slots(case).items())
        return {"bytes": float(px * 12 + sum(cat.asset(i).device_bytes() for i in range(len(cat)))),
                "flops": 60.0 * px}
    if k == "replay":
        wl = _workload("furnished", case["scenes"], case["envs"], case["width"], case["height"])
        px = case["envs"] * case["width"] * case["height"]
        return {"bytes": float(px * 8 + wl.geometry_bytes()), "flops": 60.0 * px}
    if k == "noise":
        if case["layout"] == "ragged":
            px = int((_noise_layout(case)[:, 2] * _noise_layout(case)[:, 3]).sum())
        else:
            px = case["images"] * case["width"] * case["height"]
        # One of four input pixels is sampled.
        return {"bytes": 5.0 * px, "flops": 30.0 * px}
    px = float(case["width"] * case["height"])
    if k == "occlusion":
        return {"bytes": 12.0 * px, "flops": 32 * 40 * px}
    return {"bytes": 8.0 * px, "flops": 2.0 * px}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    k = case["kind"]
    if k == "draw":
        return _exact_draw(case, seed)
    if k == "replay":
        return _exact_replay(case, seed)
    if k == "noise":
        return _exact_noise(case, seed)
    if k == "unproject":
        window = _unproject_input(case, seed).double()
        a, b = (float(v) for v in _unprojection())
        depth = window[:, :case["width"]]
        window[:, :case["width"]] = torch.where(depth == 1.0, 0.0, b / (depth + a))
        return window
    return None  # bytes, or images of many large scenes


def _triangles(wl, scene):
    """World-space triangles of one scene, [n, 3, 3] in 64 bits."""
    views = dict(wl.templates)
    out = []
    for template, bake, _ in wl.instances[scene]:
        m = np.eye(4) if bake is None else np.asarray(bake, np.float64)
        for mesh, offset, count, _ in views[template]:
            p = wl.meshes[mesh]["positions"].astype(np.float64)
            t = wl.meshes[mesh]["indices"][offset:offset + count].reshape(-1, 3)
            out.append((p @ m[:3, :3] + m[3, :3])[t])
    return torch.from_numpy(np.concatenate(out)).cuda()


def _cast(triangles, projection, view, w, h):
    """(metres, window depth) of the nearest front face at every pixel centre,
    row 0 at the bottom, by homogeneous edge functions."""
    p = torch.from_numpy(projection.astype(np.float64)).cuda()
    v = torch.from_numpy(view.astype(np.float64)).cuda()
    eye = triangles @ v[:3, :3] + v[3, :3]
    clip = eye @ p[:3] + p[3]
    lim = clip[..., 3:]
    xyz = clip[..., :3]
    x, y, q = clip[..., 0], clip[..., 1], clip[..., 3]
    a, b = [1, 2, 0], [2, 0, 1]
    edge = torch.stack([y[:, a] * q[:, b] - q[:, a] * y[:, b], q[:, a] * x[:, b] - x[:, a] * q[:, b],
                        x[:, a] * y[:, b] - y[:, a] * x[:, b]], -1)
    det = edge[:, 0, 0] * x[:, 0] + edge[:, 0, 1] * y[:, 0] + edge[:, 0, 2] * q[:, 0]
    keep = (det > 0) & ~((xyz > lim).all(1).any(1) | (xyz < -lim).all(1).any(1))
    edge, clip, eye = edge[keep], clip[keep], eye[keep]
    px = ((torch.arange(w, device="cuda", dtype=torch.float64) * 2 + 1 - w) / w).repeat(h)
    py = ((torch.arange(h, device="cuda", dtype=torch.float64) * 2 + 1 - h) / h).repeat_interleave(w)
    at = torch.stack([px, py, torch.ones_like(px)])
    best = torch.full((w * h,), math.inf, device="cuda", dtype=torch.float64)
    metres = torch.zeros(w * h, device="cuda", dtype=torch.float64)
    step = max(1, (1 << 25) // (w * h))
    for i in range(0, len(edge), step):
        e, c = edge[i:i + step], clip[i:i + step]
        l = [e[:, k] @ at for k in range(3)]
        s = l[0] + l[1] + l[2]
        zc = (l[0] * c[:, 0, 2:3] + l[1] * c[:, 1, 2:3] + l[2] * c[:, 2, 2:3]) / s
        qc = (l[0] * c[:, 0, 3:] + l[1] * c[:, 1, 3:] + l[2] * c[:, 2, 3:]) / s
        inside = (l[0] >= 0) & (l[1] >= 0) & (l[2] >= 0) & (s > 0) & (zc >= -qc) & (zc < qc)
        z = torch.where(inside, zc / qc, math.inf)
        z, who = z.min(0)
        d = eye[i:i + step, :, 2]
        own = torch.arange(w * h, device="cuda")
        m = -sum(l[k][who, own] * d[who, k] for k in range(3)) / s[who, own]
        nearer = z < best
        best = torch.where(nearer, z, best)
        metres = torch.where(nearer, m, metres)
    window = torch.where(best.isinf(), 1.0, best * 0.5 + 0.5)
    return metres.reshape(h, w), window.reshape(h, w)


def _cast_all(wl, projections, views):
    """Per environment (metres, window depth), or None when it would take long."""
    pairs = sum(float(t) * w * h for t, (w, h) in zip(wl.triangles_per_env(), wl.viewports))
    if pairs > 3e11:
        return None
    scenes = {}
    out = []
    for e, (w, h) in enumerate(wl.viewports):
        k = int(wl.scene_of_env[e])
        if k not in scenes:
            scenes[k] = _triangles(wl, k)
        out.append(_cast(scenes[k], projections[e], views[e], w, h))
    return out


def _exact_draw(case, seed):
    wl = _case_workload(case)
    projections, views = _poses(wl, seed)
    images = _cast_all(wl, projections, views)
    if images is None:
        return None
    planes = []
    for k, empty in ((0, 0.0), (1, 1.0)):
        if wl.uniform:
            w, h = wl.viewports[0]
            tx, ty = procedural.grid_for(wl.envs)
            plane = torch.full((ty * h, tx * w), empty, dtype=torch.float64, device="cuda")
            for e, image in enumerate(images):
                y, x = e // tx * h, e % tx * w
                plane[y:y + h, x:x + w] = image[k]
        else:
            plane = torch.cat([image[k].reshape(-1) for image in images])[None]
        planes.append(plane)
    out = {"color": None, "linear": planes[0], "semantic": None}
    if case["envs"] == 1:
        out["depth"] = planes[1]
    return out


def _exact_replay(case, seed):
    wl = _workload("furnished", case["scenes"], case["envs"], case["width"], case["height"])
    projections, views = _poses(wl, seed)
    images = _cast_all(wl, projections, views)
    return None if images is None else {"color": None, "depth": torch.stack([i[0] for i in images])}


def _philox(counter, key):
    """Philox4x32-10 (Salmon et al., SC'11) of uint64 arrays holding 32-bit words."""
    low = np.uint64(0xFFFFFFFF)
    c, k0, k1 = list(counter), key & 0xFFFFFFFF, key >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & low,
             (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _exact_noise_image(depth, image, seed, model, table):
    """The noise model on one image (the first call of a model with that seed)."""
    h, w = depth.shape
    idx = np.arange(h * w, dtype=np.uint64)
    z = np.zeros_like(idx)
    n = []
    for word in _philox([idx, z + np.uint64(image), z, z], seed)[:3]:
        u = (word >> np.uint64(8)).astype(np.int64)
        k, f = u >> 12, (u & 4095) / 4096.0
        n.append((table[k] + f * (table[k + 1] - table[k])).reshape(h, w))
    r, c = np.mgrid[0:h, 0:w]
    y = (np.clip(r + n[0] * 0.25, 0, h - 1) + 0.5).astype(np.int64)
    x = (np.clip(c + n[1] * 0.25, 0, w - 1) + 0.5).astype(np.int64)
    d = depth[y - y % 2, x - x % 2]
    ux = (x / max(w - 1, 1) * 639.0 + 0.5).astype(np.int64)
    uy = (y / max(h - 1, 1) * 479.0 + 0.5).astype(np.int64)
    near = np.where(d >= 10.0, 0.0, d)
    i2 = ((near + 1.0) * 0.5).astype(np.int64)
    wt = (near - ((i2 - 1) * 2.0 + 1.0)) * 0.5
    cell = (uy // 6) * 80 + ux // 8
    f = (1.0 - wt) * model[cell, np.clip(i2 - 1, 0, 4)] + wt * model[cell, np.clip(i2, 0, 4)]
    ud = np.where(f < 1e-5, 0.0, near / np.where(f < 1e-5, 1.0, f))
    q = (35.130 / np.where(ud == 0, 1.0, ud) + n[2] * 0.027778) * 8.0
    q = np.sign(q) * np.floor(np.abs(q) + 0.5)
    ok = (d < 10.0) & (ud != 0) & (q > 1e-5)
    return np.where(ok, 35.130 * 8.0 / np.where(ok, q, 1.0), 0.0)


def _exact_noise(case, seed):
    depth = _noise_input(case, seed).double().cpu().numpy()
    model = noise.load_model().astype(np.float64).reshape(-1, 5)
    knots = (torch.arange(4097, dtype=torch.float64) + 0.5) / 4097.0
    table = torch.special.ndtri(knots).numpy()
    if case["layout"] == "one":
        return _exact_noise_image(depth, 0, seed, model, table)
    out = np.zeros_like(depth)
    w, h = case["width"], case["height"]
    tx = procedural.grid_for(case["images"])[0]
    for i in range(case["images"]):
        if case["layout"] == "tiles":
            at = (slice(i // tx * h, i // tx * h + h), slice(i % tx * w, i % tx * w + w))
            out[at] = _exact_noise_image(depth[at], i, seed, model, table)
        else:
            o, _, iw, ih = (int(v) for v in _noise_layout(case)[i])
            image = _exact_noise_image(depth[o:o + iw * ih].reshape(ih, iw), i, seed, model, table)
            out[o:o + iw * ih] = image.reshape(-1)
    return out
