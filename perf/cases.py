"""Performance cases of the renderer: what users of this framework have it do, through its public entry points.

A case is a dict of plain values; `kind` says which entry points it calls:

  frame    BDPTRenderer.render: one frame into a host image (C1, textured, mixed and three-light scenes under point
           lights; the 64-object scene under an HDRI sky, with either estimator)
  batch    BatchRenderer.render of a material sweep: jobs of uneven size, samples and material set, then development
  adjoint  MaterialRenderer.image, an image loss and its backward pass (path replay)
  fit      one step of the batched inverse fit: set materials, forward batch, image loss, adjoint batch
  create   RenderScene: commit a scene (upload, acceleration structure), then the first queries against it
  trace    RenderScene.trace: closest hits of a host array of rays
  develop  post.develop, the median denoiser and the 8-bit conversion of a film on the device

Geometry, textures and skies are the repository's own synthetic scenes; a seed draws what differs between two uses of
such a scene: the view, the materials, the lights' place and power, and the random streams.
"""
import ctypes as C
import dataclasses
import functools
import importlib
import math

import numpy as np
import torch

omv = importlib.import_module("openmaterial-validation_gb300")
diff = importlib.import_module("openmaterial-validation_gb300.diff")
post = importlib.import_module("openmaterial-validation_gb300.post")
S = omv.scenes

# Rays per path of each scene family (camera extension, connection, light), rounded from the renderer's ray counters.
RAYS = {"c1": (1.6, 0.5, 1.0), "lights": (1.6, 0.5, 1.0), "mixed": (2.0, 0.8, 1.2), "textured": (2.0, 0.8, 1.2),
        "materials": (2.0, 0.8, 1.1), "c2": (1.2, 0.0, 0.0)}
LIT = ("c1", "lights", "mixed", "textured", "materials")


def listed():
    return [
        # an interactive preview: the smallest frame, all launches and latency
        {"name": "preview_c1_64x64x1", "kind": "frame", "scene": "c1", "w": 64, "h": 64, "spp": 1, "mis": False},
        # the point-light configuration at its own size
        {"name": "frame_c1_256x256x16", "kind": "frame", "scene": "c1", "w": 256, "h": 256, "spp": 16, "mis": False},
        # the same scene as a final full-HD frame
        {"name": "frame_c1_1920x1080x64", "kind": "frame", "scene": "c1", "w": 1920, "h": 1080, "spp": 64, "mis": False},
        # the headline frame: a million triangles in 64 instances under a sky
        {"name": "frame_c2_1920x1080x64", "kind": "frame", "scene": "c2", "tri_scale": 1.0, "w": 1920, "h": 1080, "spp": 64,
         "mis": False},
        # textures, normal maps, masked and blended materials at an odd size
        {"name": "frame_textured_641x479x17", "kind": "frame", "scene": "textured", "w": 641, "h": 479, "spp": 17, "mis": False},
        # the estimator users pick for bright suns
        {"name": "mis_c2_960x540x16", "kind": "frame", "scene": "c2", "tri_scale": 1.0, "w": 960, "h": 540, "spp": 16, "mis": True},
        # a material sweep: many jobs of uneven size in one call
        {"name": "batch_16_jobs", "kind": "batch", "jobs": 16, "tris": 200_000, "side_lo": 128, "side_hi": 512, "spp_lo": 4,
         "spp_hi": 32, "graph": True},
        # the gradient configuration: forward and backward of an image loss
        {"name": "adjoint_512x512x32", "kind": "adjoint", "tris": 100_000, "materials": 8, "w": 512, "h": 512, "spp": 32},
        # one optimisation step of the inverse fit over a group of scenes
        {"name": "fit_8_scenes_128x128x16", "kind": "fit", "scenes": 8, "tris": 20_000, "side": 128, "spp": 16},
        # loading a scene: commit and the first picks
        {"name": "create_c2_1m", "kind": "create", "tri_scale": 1.0, "rays": 4096},
        # batched visibility queries from a host program
        {"name": "trace_200k_tris_1m_rays", "kind": "trace", "tris": 200_000, "rays": 1_000_000},
        # image development of a full-HD film
        {"name": "develop_1920x1080", "kind": "develop", "w": 1920, "h": 1080, "half": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "batch", "adjoint", "fit", "create", "trace", "develop"])
    if kind == "frame":
        sky = rng.random() < 0.4
        scene = "c2" if sky else rng.choice(LIT)
        mis = sky and rng.random() < 0.4
        w = _log_int(rng, 64, 1920)
        h = max(36, int(w * rng.uniform(0.5, 1.0)))
        h = min(h, 1080)
        # at most the listed frames' cost: full HD at 64 samples for the cheap scenes, less for the others
        most = 130e6 if scene in ("c1", "c2") and not mis else 40e6
        spp = _log_int(rng, 1, max(1, min(64, most / (w * h))))
        case = {"kind": "frame", "scene": scene, "w": w, "h": h, "spp": spp, "mis": mis}
        if sky:
            case["tri_scale"] = rng.choice([1.0, 0.25, 0.06])
        return case
    if kind == "batch":
        lo = _log_int(rng, 32, 200)
        hi = lo + _log_int(rng, 16, 300)
        return {"kind": "batch", "jobs": rng.randint(3, 16), "tris": _log_int(rng, 5_000, 200_000), "side_lo": lo, "side_hi": hi,
                "spp_lo": rng.randint(1, 4), "spp_hi": rng.randint(5, 32), "graph": rng.random() < 0.5}
    if kind == "adjoint":
        w = _log_int(rng, 48, 500)
        h = _log_int(rng, 48, 500)
        return {"kind": "adjoint", "tris": _log_int(rng, 5_000, 100_000), "materials": rng.choice([4, 6, 8]), "w": w, "h": h,
                "spp": _log_int(rng, 2, 30)}
    if kind == "fit":
        return {"kind": "fit", "scenes": rng.randint(2, 8), "tris": _log_int(rng, 5_000, 50_000), "side": _log_int(rng, 40, 160),
                "spp": _log_int(rng, 4, 16)}
    if kind == "create":
        return {"kind": "create", "tri_scale": rng.uniform(0.02, 0.95), "rays": _log_int(rng, 256, 20_000)}
    if kind == "trace":
        return {"kind": "trace", "tris": _log_int(rng, 2_000, 200_000), "rays": _log_int(rng, 300, 1_000_000)}
    w = _log_int(rng, 100, 1920)
    return {"kind": "develop", "w": w, "h": max(3, int(w * rng.uniform(0.4, 0.56))), "half": rng.choice([1, 1, 2])}


# ---------------------------------------------------------------- scenes ---

@functools.lru_cache(maxsize=4)
def _sky_scene(tri_scale):
    """The 64-object scene's geometry and sky (assets that a program loads once)."""
    return S.scene_c2(64, 64, 1, tri_scale=tri_scale, sky_size=(2048, 1024) if tri_scale >= 1.0 else (512, 256))


@functools.lru_cache(maxsize=4)
def _material_scene(tris, n_materials, seed, sky):
    return S.scene_materials(64, 64, 1, tris=tris, n_materials=n_materials, seed=seed, sky=sky)


@functools.lru_cache(maxsize=1)
def _textured_scene():
    return S.scene_textured(64, 64, 1)


def _spec(case, rng):
    """The scene of a frame or create case, with the seed's view, materials and lights."""
    w, h, spp = case.get("w", 64), case.get("h", 64), case.get("spp", 1)
    name = case.get("scene", "c2")
    if name == "c2":
        base = _sky_scene(case["tri_scale"])
        mats = [dataclasses.replace(m, base_color=tuple(float(x) for x in rng.uniform(0, 1, 3)) + (1.0,),
                                    roughness=float(rng.uniform(0.05, 1.0)), metallic=float(rng.integers(0, 2)))
                for m in base.materials]
        cam = S.camera_default(w, h)
        yaw, pitch = rng.uniform(-math.pi, math.pi), rng.uniform(-0.3, 0.3)
        cam.rotation = S.default_view((0.0, 0.0, 0.0), (math.sin(yaw) * math.cos(pitch), math.sin(pitch), -math.cos(yaw) * math.cos(pitch)))
        return dataclasses.replace(base, materials=mats, camera=cam, render=dataclasses.replace(base.render, samples_per_pixel=spp))
    if name == "materials":
        base = _material_scene(50_000, 8, 0, False)
    elif name == "textured":
        base = _textured_scene()
    else:
        base = {"c1": S.scene_c1, "lights": S.scene_lights, "mixed": S.scene_mixed}[name](w, h, spp)
    lights = [dataclasses.replace(lt, position=tuple(float(p + d) for p, d in zip(lt.position, rng.uniform(-0.5, 0.5, 3))),
                                  intensity=tuple(float(i * f) for i, f in zip(lt.intensity, rng.uniform(0.7, 1.4, 3))))
              for lt in base.lights]
    focus = (h / 2.0) / math.tan(math.radians(22.5))
    cam = S.camera_from_json(w, h, w / h, focus, 45.0, position=tuple(float(x) for x in np.asarray(base.camera.position) + rng.uniform(-0.1, 0.1, 3)))
    return dataclasses.replace(base, lights=lights, camera=cam, render=dataclasses.replace(base.render, samples_per_pixel=spp))


def _triangles(case):
    kind = case["kind"]
    if kind in ("frame", "create"):
        if case.get("scene", "c2") == "c2":
            return 1_048_576 * case["tri_scale"]
        return {"c1": 5_122, "lights": 5_122, "mixed": 1_602, "textured": 1_602, "materials": 50_000}[case["scene"]]
    return case["tris"] * case.get("scenes", 1)


def _square_camera(spec_camera, side):
    cam = omv.PinholeCamera.from_spec(spec_camera)
    cam.width = cam.height = side
    cam.adjust_to_resolution()
    cam.set_y_fov(45.0)
    return cam


def _film(h, w):
    return (torch.zeros((h, w, 3), dtype=torch.float64, device="cuda"), None, torch.zeros((h, w), dtype=torch.int32, device="cuda"))


def _batch_sizes(case):
    """The sweep's resolutions and samples: the same for every seed of a case."""
    rng = np.random.default_rng([case["jobs"], case["side_lo"], case["side_hi"], case["spp_lo"], case["spp_hi"]])
    return (rng.integers(case["side_lo"], case["side_hi"] + 1, case["jobs"]),
            rng.integers(case["spp_lo"], case["spp_hi"] + 1, case["jobs"]))


def _trace_rays(case, seed):
    """Rays as a program that asks for visibility has them: half from one viewpoint, half between random points."""
    rng = np.random.default_rng([seed, 2])
    n = case["rays"]
    r = np.zeros((n, 8), dtype=np.float32)
    a = n // 2
    target = rng.uniform((-4.0, -1.0, -8.0), (4.0, 1.5, -2.0), (n, 3))
    org = np.broadcast_to(np.array([0.0, 1.5, 4.0]) + rng.uniform(-0.2, 0.2, 3), (n, 3)).copy()
    org[a:] = rng.uniform((-5.0, 0.5, -10.0), (5.0, 4.0, 3.0), (n - a, 3))
    d = target - org
    r[:, 0:3] = org
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 7] = 3.0e38
    return r


# --------------------------------------------------------------- prepare ---

def prepare(case, seed):
    omv.build()
    rng = np.random.default_rng([seed, 0])
    kind = case["kind"]
    if kind == "frame":
        spec = _spec(case, rng)
        renderer = omv.BDPTRenderer()
        renderer.set_scene(omv.RenderScene(spec))
        renderer.set_parameters(omv.RendererParameters.for_scene(
            spec, seed=seed, estimator=omv.ESTIMATOR_MIS if case["mis"] else omv.ESTIMATOR_REFERENCE))
        return {"kind": kind, "renderer": renderer, "camera": omv.PinholeCamera.from_spec(spec.camera)}
    if kind == "batch":
        spec = _material_scene(case["tris"], 8, 0, False)
        rs = omv.RenderScene(spec)
        br = omv.BatchRenderer(rs, omv.RendererParameters.for_scene(spec))
        br.set_material_sets(S.material_variants(spec, case["jobs"], seed=seed))
        sides, spps = _batch_sizes(case)
        films = [_film(int(s), int(s)) for s in sides]
        jobs = [br.job(_square_camera(spec.camera, int(s)), int(n), f, seed=1000 * (seed % 10_000) + j, material_set=j)
                for j, (s, n, f) in enumerate(zip(sides, spps, films))]
        return {"kind": kind, "batch": br, "films": films, "jobs": jobs, "graph": case["graph"]}
    if kind == "adjoint":
        base = _material_scene(case["tris"], case["materials"], 0, False)
        focus = (case["h"] / 2.0) / math.tan(math.radians(22.5))
        cam = S.camera_from_json(case["w"], case["h"], case["w"] / case["h"], focus, 45.0, position=base.camera.position)
        spec = dataclasses.replace(base, camera=cam, materials=S.material_variants(base, 1, seed=seed)[0])
        R = diff.MaterialRenderer(spec, spp=case["spp"], seed=2 * seed + 1, adjoint_seed=2 * seed + 2)
        P = torch.tensor(diff.params_from_materials(spec.materials), dtype=torch.float64, requires_grad=True)
        g = torch.Generator(device="cuda").manual_seed(seed)
        target = torch.rand((case["h"], case["w"], 3), dtype=torch.float64, device="cuda", generator=g)
        return {"kind": kind, "renderer": R, "params": P, "target": target}
    if kind == "fit":
        n, side = case["scenes"], case["side"]
        scs = [_material_scene(case["tris"], 4, 100 + j, True) for j in range(n)]
        scs = [dataclasses.replace(sc, hdri=scs[0].hdri, materials=S.material_variants(sc, 1, seed=seed + j)[0]) for j, sc in enumerate(scs)]
        group = omv.RenderScene.group(scs)
        br = omv.BatchRenderer(group, omv.RendererParameters.for_scene(scs[0], samplesPerPixel=case["spp"]))
        films = [_film(side, side) for _ in scs]
        cams = [_square_camera(sc.camera, side) for sc in scs]
        base = 1000 * (seed % 10_000)
        fwd = [br.job(cams[j], case["spp"], films[j], seed=base + 2 * j + 1, part=j) for j in range(n)]
        bwd = [br.job(cams[j], case["spp"], films[j], seed=base + 2 * j + 2, part=j) for j in range(n)]
        g = torch.Generator(device="cuda").manual_seed(seed)
        targets = [torch.rand((side, side, 3), dtype=torch.float32, device="cuda", generator=g) for _ in scs]
        grads = [torch.zeros((len(sc.materials), diff.SLOTS), dtype=torch.float32, device="cuda") for sc in scs]
        return {"kind": kind, "group": group, "batch": br, "scenes": scs, "films": films, "fwd": fwd, "bwd": bwd,
                "targets": targets, "grads": grads, "params": [diff.params_from_materials(sc.materials) for sc in scs]}
    if kind == "create":
        spec = _spec(case, rng)
        n = case["rays"]
        rays = np.zeros((n, 8), dtype=np.float32)
        d = rng.normal(size=(n, 3))
        rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
        rays[:, 7] = 3.0e38
        return {"kind": kind, "spec": spec, "rays": rays}
    if kind == "trace":
        return {"kind": kind, "scene": omv.RenderScene(_material_scene(case["tris"], 8, 0, False)), "rays": _trace_rays(case, seed)}
    return {"kind": kind, "half": case["half"], **_develop_inputs(case, seed)}


def _develop_inputs(case, seed):
    """A film of about 64 samples per pixel: log-normal radiance with a few very bright pixels and some never hit."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    h, w = case["h"], case["w"]
    count = torch.randint(1, 65, (h, w), dtype=torch.int32, device="cuda", generator=g)
    x = torch.randn((h, w, 3), dtype=torch.float64, device="cuda", generator=g).mul_(1.2).sub_(1.0).exp_()
    u = torch.rand((h, w, 1), dtype=torch.float64, device="cuda", generator=g)
    x = torch.where(u < 0.001, x * 1e4, x)
    count = torch.where(u[..., 0] > 0.999, torch.zeros_like(count), count)
    return {"sum": (x * count.unsqueeze(-1)).contiguous(), "count": count.contiguous()}


# ------------------------------------------------------------------- run ---

def _hits(h):
    return {k: h[k] for k in ("inst", "geom", "prim", "material", "t", "u", "v")}


def run(s):
    kind = s["kind"]
    if kind == "frame":
        return s["renderer"].render(s["camera"])
    if kind == "batch":
        for f in s["films"]:
            f[0].zero_()
            f[2].zero_()
        s["batch"].render(s["jobs"], graph=s["graph"])
        return [post.develop(f[0], f[2], tonemapped=False, rgba8=False)["linear"] for f in s["films"]]
    if kind == "adjoint":
        P = s["params"]
        P.grad = None
        image = s["renderer"].image(P)
        loss = ((image - s["target"]) ** 2).mean()
        loss.backward()
        return {"image": image.detach().float(), "grad": P.grad.float()}
    if kind == "fit":
        return _fit_step(s)
    if kind == "create":
        scene = omv.RenderScene(s["spec"])
        lo, hi = scene.bounds()
        return {**_hits(scene.trace(s["rays"])), "lo": lo, "hi": hi}
    if kind == "trace":
        return _hits(s["scene"].trace(s["rays"]))
    out = post.develop(s["sum"], s["count"])
    clean = post.SimpleDenoiserMedian(out["tonemapped"], s["half"])
    return {**out, "denoised": clean, "denoised8": post.rgba8(clean, flip=True)}


def _fit_step(s):
    """One step as the inverse fit makes it: materials, forward batch, squared error, adjoint batch."""
    mats, keep = [], []
    for sc, P in zip(s["scenes"], s["params"]):
        mats += diff.materials_from_params(sc.materials, P)
    descs = omv.capi.material_descs(mats, keep)
    omv.check(omv.lib().omv_scene_set_materials(s["group"].handle, len(mats), descs))
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for f in s["films"]:
        f[0].zero_()
        f[2].zero_()
    s["batch"].render(s["fwd"], stream)
    images = [post.develop(f[0], f[2], tonemapped=False, rgba8=False)["linear"] for f in s["films"]]
    adjoints = [((2.0 / t.numel()) * (i[..., :3] - t)).contiguous() for i, t in zip(images, s["targets"])]
    for g in s["grads"]:
        g.zero_()
    s["batch"].adjoint(s["bwd"], adjoints, s["grads"], stream)
    torch.cuda.synchronize()
    return {"images": images, "grads": s["grads"]}


# ------------------------------------------------------------------ work ---

def work(case):
    """Bytes: the scene once and the results once.  Operations: for each ray one path through an 8-wide tree (8 boxes of
    about 12 operations a level) and one triangle, for each vertex its shading; rays per path from the ray counters."""
    kind = case["kind"]
    if kind == "develop":
        n = case["w"] * case["h"]
        # film read; linear, tone-mapped and 8-bit images written; the median reads and writes an image, then 8-bit again
        return {"bytes": n * (28 + 36 + 32 + 20), "flops": n * (30 + 6 * 19 * (1 if case["half"] == 1 else 8))}
    tris = _triangles(case)
    scene_bytes = tris * (48 + 12 + 24)
    per_ray = 96 * (2 + math.log(max(8.0, tris), 8)) + 60
    if kind == "create":
        return {"bytes": tris * (12 + 18 + 48 + 12 + 24 + 24), "flops": tris * 20 * math.log2(max(2.0, tris)) + case["rays"] * per_ray}
    if kind == "trace":
        return {"bytes": scene_bytes + case["rays"] * (32 + 32), "flops": case["rays"] * per_ray}
    if kind == "frame":
        family, pixels = case["scene"], case["w"] * case["h"]
        paths = pixels * case["spp"]
    elif kind == "batch":
        family = "materials"
        pixels = case["jobs"] * ((case["side_lo"] + case["side_hi"]) / 2) ** 2
        paths = pixels * (case["spp_lo"] + case["spp_hi"]) / 2
    else:
        family = "materials"
        pixels = case["w"] * case["h"] if kind == "adjoint" else case["scenes"] * case["side"] ** 2
        paths = 2 * pixels * case["spp"]  # forward and replay
    ext, conn, light = RAYS[family]
    vertices = ext + light
    if case.get("mis"):
        conn += ext
    return {"bytes": scene_bytes + 16 * pixels, "flops": paths * ((ext + conn + light) * per_ray + 300 * vertices)}


# ----------------------------------------------------------------- exact ---

def exact(case, seed):
    """Values in 64 bits where plain torch can give them: development, and closest hits of small queries.  A rendered
    image, its gradients and a scene's boxes have none (millions of random paths)."""
    if case["kind"] == "develop":
        return _exact_develop(case, seed)
    if case["kind"] == "trace" and case["rays"] * case["tris"] <= 4e9:
        return _exact_trace(case, seed)
    return None


def _exact_develop(case, seed):
    s = _develop_inputs(case, seed)
    n = s["count"].double().clamp(min=1.0).unsqueeze(-1)
    rgb = torch.where(s["count"].unsqueeze(-1) > 0, s["sum"] / n, s["sum"])
    one = torch.ones_like(rgb[..., :1])
    lum = rgb @ torch.tensor([0.2126, 0.7152, 0.0722], dtype=torch.float64, device=rgb.device)
    scale = torch.where(lum > torch.finfo(torch.float32).eps, lum.clamp(min=1e-300) ** -0.5, torch.ones_like(lum))
    tone = (rgb * scale.unsqueeze(-1)).clamp(0.0, 1.0)
    h, w, r = case["h"], case["w"], case["half"]
    clean = tone.clone()
    if h > 2 * r and w > 2 * r:
        k = 2 * r + 1
        win = torch.stack([tone[dy:h - 2 * r + dy, dx:w - 2 * r + dx] for dy in range(k) for dx in range(k)])
        clean[r:h - r, r:w - r] = win.median(dim=0).values
    cat = lambda x: torch.cat([x, one], dim=-1)  # noqa: E731
    return {"linear": cat(rgb), "tonemapped": cat(tone), "rgba8": None, "denoised": cat(clean), "denoised8": None}


def _exact_trace(case, seed):
    """Moeller-Trumbore over all triangles in 64 bits."""
    spec = _material_scene(case["tris"], 8, 0, False)
    world = []
    for inst in spec.instances:
        m = spec.meshes[inst.mesh]
        p = m.positions.astype(np.float64) @ inst.transform[:3, :3].astype(np.float64).T + inst.transform[:3, 3].astype(np.float64)
        world.append(p[m.faces.astype(np.int64)])
    tri = torch.from_numpy(np.concatenate(world)).cuda()
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    rays = torch.from_numpy(_trace_rays(case, seed)).cuda().double()
    t_all, u_all, v_all = [], [], []
    # with o and d expanded, every term is a product of one matrix of rays and one of triangles
    n = torch.linalg.cross(e1, e2)
    an, ae1, ae2 = (a * n).sum(1), torch.linalg.cross(a, e1), torch.linalg.cross(a, e2)
    for r in rays.split(max(1, 40_000_000 // len(tri))):
        o, d = r[:, 0:3], r[:, 4:7]
        od = torch.linalg.cross(o, d)
        det = -(d @ n.T)
        # u = (o - a) . (d x e2) / det, v = (o - a) . (e1 x d) / det, t = (o - a) . n / det
        u = (od @ e2.T + d @ ae2.T) / det
        v = -(od @ e1.T + d @ ae1.T) / det
        t = (o @ n.T - an) / det
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 0)
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        best, at = t.min(dim=1)
        hit = torch.isfinite(best)
        zero = torch.zeros_like(best)
        t_all.append(torch.where(hit, best, zero))
        u_all.append(torch.where(hit, u.gather(1, at[:, None])[:, 0], zero))
        v_all.append(torch.where(hit, v.gather(1, at[:, None])[:, 0], zero))
    cat = lambda x: torch.cat(x).cpu().numpy()  # noqa: E731
    return {"inst": None, "geom": None, "prim": None, "material": None, "t": cat(t_all), "u": cat(u_all), "v": cat(v_all)}
