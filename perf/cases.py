"""What a user of the framework has it do, as measurable passes through its public entry points.

Each case is one call a host program makes: a ray query batch (device tensors or host arrays), a
mesh rebuilt and traced (moving geometry), a query through instances, a rendered image read back, a
radiance-cache evaluation. Sizes are those of the repository's workloads (the 1M-triangle soup and
its 16M rays, 1080p camera rays, the 32 x 32 instanced grid, the 256 x 256 spectral Cornell box, the
287-slot OPENPBR grid scene, 65,536 cache records), its tests' small meshes, and ranges around them.

The scenes' colour and energy tables are smooth analytic stand-ins, handed over the way a host
without the licensed data files would: multi-lobe fits of the colour-matching functions (Wyman,
Sloan and Shirley 2013), a 6504 K Planckian illuminant, and closed-form energy tables.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import metal_vibe_tracer_b200 as vt
from metal_vibe_tracer_b200 import _lib, nrc, scenes
from metal_vibe_tracer_b200.accel import instances_array

DEV = "cuda:0"


# ---- the cases --------------------------------------------------------------------------------------
def listed():
    return [
        # A picking or probe query: a small mesh, a few thousand rays; launch latency counts.
        {"name": "pick_small", "kind": "trace", "faces": 20_000, "rays": 4_096, "set": "random", "query": "closest"},
        # The traversal microbenchmark's headline set: 1M-triangle soup, 16M incoherent rays.
        {"name": "closest_incoherent_16m", "kind": "trace", "faces": 1_000_000, "rays": 1 << 24, "set": "random",
         "query": "closest"},
        # Shadow rays of a 1080p frame: any-hit on coherent rays.
        {"name": "shadow_1080p", "kind": "trace", "faces": 1_000_000, "rays": 1920 * 1080, "set": "camera",
         "query": "any"},
        # A host renderer's ray batch in ordinary (pageable) arrays, an odd count.
        {"name": "host_batch", "kind": "host", "faces": 200_000, "rays": 1_000_003, "query": "closest"},
        # Moving geometry, small: one displaced sphere rebuilt and a preview frame traced.
        {"name": "rebuild_small", "kind": "rebuild", "faces": 20_480, "width": 320, "height": 200, "leaf": 2},
        # Moving geometry, large: the 1M-triangle soup rebuilt and a 1080p frame traced.
        {"name": "rebuild_1m", "kind": "rebuild", "faces": 1_000_000, "width": 1920, "height": 1080, "leaf": 2},
        # Instances: the 32 x 32 grid of displaced subdivision-5 icospheres through two levels.
        {"name": "instances_32x32", "kind": "instances", "grid": 32, "subdivisions": 5, "rays": 1 << 20, "query": "closest"},
        # The smallest render call: one sample of an RGB preview through the default integrator.
        {"name": "preview_64", "kind": "render", "scene": "cornell", "width": 64, "height": 64, "spp": 1, "depth": 5,
         "spectral": False, "sampler": 0, "path": "megakernel"},
        # The spectral Cornell box of the headline path-tracing workload.
        {"name": "cornell_spectral", "kind": "render", "scene": "cornell", "width": 256, "height": 256, "spp": 16,
         "depth": 8, "spectral": True, "sampler": 0, "path": "wavefront"},
        # Production rendering: OPENPBR slots with thin films, a light tree, spectral, 1080p, depth 12.
        {"name": "production_1080p", "kind": "render", "scene": "production", "width": 1920, "height": 1080, "spp": 4,
         "depth": 12, "spectral": True, "sampler": 0, "path": "wavefront"},
        # ReSTIR DI + GI frames (sampling mode 0) of a Lambert scene lit by emitter triangles; ragged.
        {"name": "restir_frames", "kind": "render", "scene": "lambert", "width": 1001, "height": 563, "spp": 4,
         "depth": 6, "spectral": False, "sampler": 1, "path": "restir"},
        # The radiance cache: the loss gradients of one frame's 65,536 training records and a cached
        # frame of the Cornell box (paths end in the network's predictions).
        {"name": "cache_frame", "kind": "cache", "records": 65_536, "levels": 16, "log2_table": 15, "spectral": True,
         "width": 512, "height": 512, "spp": 4, "depth": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "trace", "host", "rebuild", "rebuild", "instances", "render", "render", "render",
                       "cache"])
    if kind == "trace":
        return {"kind": kind, "faces": _log(rng, 500, 1_000_000), "rays": _log(rng, 1_000, 1 << 24),
                "set": rng.choice(["random", "camera"]), "query": rng.choice(["closest", "any"])}
    if kind == "host":
        return {"kind": kind, "faces": _log(rng, 5_000, 500_000), "rays": _log(rng, 10_000, 4_000_000),
                "query": rng.choice(["closest", "any"])}
    if kind == "rebuild":
        w = rng.choice([160, 320, 640, 1279, 1920])
        return {"kind": kind, "faces": _log(rng, 1_000, 1_000_000), "width": w, "height": (w * 9) // 16,
                "leaf": rng.choice([1, 2, 2, 4, 8])}
    if kind == "instances":
        return {"kind": kind, "grid": rng.randint(2, 32), "subdivisions": rng.randint(2, 5), "rays": _log(rng, 10_000, 1 << 20),
                "query": rng.choice(["closest", "any"])}
    if kind == "cache":
        return {"kind": kind, "records": _log(rng, 1_000, 65_536), "levels": rng.choice([8, 12, 16]),
                "log2_table": rng.choice([13, 14, 15]), "spectral": rng.random() < 0.5,
                "width": rng.randint(64, 512), "height": rng.randint(64, 512), "spp": rng.randint(1, 4), "depth": rng.choice([4, 8])}
    scene = rng.choice(["cornell", "lambert", "production"])
    path = rng.choice(["wavefront", "wavefront", "megakernel", "restir"])
    most = 400_000 if path != "wavefront" else 2_000_000
    pixels = _log(rng, 4_000, most)
    w = max(16, int(math.sqrt(pixels * rng.uniform(0.8, 2.0))))
    h = max(16, pixels // w)
    spp = max(1, min(16, int(4_000_000 * (0.25 if path != "wavefront" else 1.0) / (w * h) * rng.random())))
    return {"kind": kind, "scene": scene, "width": w, "height": h, "spp": spp, "depth": rng.choice([3, 6, 8, 12]),
            "spectral": rng.random() < 0.5, "sampler": rng.choice([0, 0, 1]), "path": path}


# ---- data a program keeps across calls -----------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _context():
    ctx = vt.Context(0)
    # The energy tables the coat and diffuse lobes read (32^3 and 32^2) and the sheen fit, closed form.
    n = 32
    ior = 1.0 + 2.0 * (np.arange(n) + 0.5) / n
    f0 = ((ior - 1) / (ior + 1)) ** 2
    alpha = ((np.arange(n) + 0.5) / n) ** 2
    cos = (np.arange(n) + 0.5) / n
    albedo = f0[:, None, None] + (1 - f0[:, None, None]) * (1 - cos[None, None, :]) ** 5 * (1 - 0.6 * alpha[None, :, None])
    energy = np.round(65535 * (1 - albedo)).astype(np.uint16)
    average = np.round(65535 * (1 - (2 * albedo * cos[None, None, :]).mean(2))).astype(np.uint16)
    ltc = np.tile(np.array([1.0, 0.0, 0.1], np.float32), n * n)
    tables = _lib.OpenPBRTables(energy.ctypes.data, average.ctypes.data, ltc.ctypes.data)
    if vt.load().vt_openpbr_tables_set(ctx.handle, tables) != _lib.VT_OK:
        raise RuntimeError("vt_openpbr_tables_set failed")
    ctx._pbr_tables_set = True
    return ctx


@functools.lru_cache(maxsize=None)
def _spectral_tables():
    def lobe(x, mu, s1, s2):
        return np.exp(-0.5 * ((x - mu) / np.where(x < mu, s1, s2)) ** 2)

    def cmf(lam):
        x = 1.056 * lobe(lam, 599.8, 37.9, 31.0) + 0.362 * lobe(lam, 442.0, 16.0, 26.7) - 0.065 * lobe(lam, 501.1, 20.4, 26.2)
        y = 0.821 * lobe(lam, 568.8, 46.9, 40.5) + 0.286 * lobe(lam, 530.9, 16.3, 31.1)
        z = 1.217 * lobe(lam, 437.0, 11.8, 36.0) + 0.681 * lobe(lam, 459.0, 26.0, 13.8)
        return np.stack([x, y, z], 1)

    def planck(lam):
        return 1.0 / (lam ** 5 * np.expm1(1.4388e7 / (lam * 6504.0)))

    m = np.array([[3.2404542, -1.5371385, -0.4985314], [-0.9692660, 1.8760108, 0.0415560], [0.0556434, -0.2040259, 1.0572252]])
    full, lam = np.arange(360, 831, dtype=np.float64), np.arange(380, 781, dtype=np.float64)
    weights = (cmf(full) @ m.T) * planck(full)[:, None]
    scale = 1.0 / weights.sum(0)                          # the illuminant maps to rgb (1, 1, 1)
    rgb = (cmf(lam) @ m.T)
    spd = planck(lam)
    spd = spd / (cmf(lam)[:, 1] * spd).sum()
    rgb = rgb / (rgb * spd[:, None]).sum(0)
    s = np.abs(rgb).sum(1)
    trapezoid = lambda v: (0.5 * (v[1:] + v[:-1])).sum()  # noqa: E731
    density = 0.9 * spd * s / trapezoid(spd * s) + 0.1 * s / trapezoid(s)
    cdf = np.concatenate([[0.0], np.cumsum(0.5 * (density[1:] + density[:-1]))])
    icdf = np.interp(np.linspace(0, 1, 1025), cdf / cdf[-1], lam)
    visible = np.cumsum(cmf(full).sum(1) + 0.01)
    phase = -math.pi + math.pi * (visible - visible[0]) / (visible[-1] - visible[0])
    return {"cmf_rgb": rgb.astype(np.float32), "illum": spd.astype(np.float32), "icdf": icdf.astype(np.float32),
            "cos_phase": np.cos(np.interp(lam, full, phase)).astype(np.float32), "uplift_w": weights * scale[None, :],
            "uplift_cos": np.cos(phase), "lambda_min": 380}


@functools.lru_cache(maxsize=4)
def _grid_scene(name):
    if name == "production":
        return scenes.production_scene(seed=0, triangles=740_000, emitters=20_000)
    return scenes.sphere_grid(300_000, seed=0, coloured=True)


@functools.lru_cache(maxsize=None)
def _asset(subdivisions, seed):
    return scenes.displaced_sphere_asset(subdivisions, seed)


def _random(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _soup(n, seed):
    """scenes.triangle_soup's distribution for n triangles in all, made on the GPU: (faces (n, 4) int32,
    vertices (3 n, 8) float32). Edge lengths keep the 1M soup's hit rates as n shrinks."""
    g = _random(seed)
    centre = torch.rand(n, 3, generator=g, device=DEV)
    edge = torch.exp(math.log(0.002 * math.sqrt(1e6 / n)) + 0.5 * torch.randn(n, 1, generator=g, device=DEV))
    a = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device=DEV), dim=1)
    b = torch.nn.functional.normalize(torch.linalg.cross(a, torch.randn(n, 3, generator=g, device=DEV)), dim=1)
    r = edge / math.sqrt(3.0)
    v = torch.zeros(n, 3, 8, device=DEV)
    for k in range(3):
        t = 2 * math.pi * k / 3
        v[:, k, :3] = centre + r * (math.cos(t) * a + math.sin(t) * b)
    f = torch.zeros(n, 4, dtype=torch.int32, device=DEV)
    f[:, :3] = torch.arange(3 * n, dtype=torch.int32, device=DEV).view(n, 3)
    return f, v.view(3 * n, 8)


def _rays(case, seed):
    n = case["rays"]
    g = _random(seed + 7)
    if case.get("set", "random") == "camera":
        w = max(1, int(math.sqrt(n * 16 / 9)))
        h = -(-n // w)
        rays = scenes.coherent_rays_torch(w, h, DEV)[:n].contiguous()
        rays[:, 0:3] += 0.02 * torch.rand(3, generator=g, device=DEV)
        span = (1.0, 2.2)
    else:
        rays = torch.empty(n, 8, device=DEV)
        rays[:, 0:3] = torch.rand(n, 3, generator=g, device=DEV)
        rays[:, 3] = 0.0
        rays[:, 4:7] = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device=DEV), dim=1)
        rays[:, 7] = math.inf
        span = (0.05, 1.0)
    if case["query"] == "any":  # shadow rays end somewhere
        rays[:, 7] = span[0] + (span[1] - span[0]) * torch.rand(n, generator=g, device=DEV)
    return rays


def _camera(seed):
    """A viewpoint over the unit cube's middle, another one per seed."""
    a = 2 * math.pi * ((seed * 0.618034) % 1.0)
    return {"pos": (0.5 + 1.7 * math.sin(a), 0.9, 0.5 + 1.7 * math.cos(a)), "target": (0.5, 0.5, 0.5), "up": (0.0, 1.0, 0.0),
            "fov": 45.0}


# ---- one state per case -----------------------------------------------------------------------------------
def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    if kind in ("trace", "host"):
        faces, verts = _soup(case["faces"], seed)
        mesh = vt.Mesh(ctx, faces, verts)
        rays = _rays(case, seed)
        if kind == "host":
            rays = rays.cpu().numpy().view(vt.RAY_DTYPE).reshape(-1)
        return {"kind": kind, "mesh": mesh, "rays": rays, "query": case["query"]}
    if kind == "rebuild":
        faces, verts = _soup(case["faces"], seed)
        return {"kind": kind, "ctx": ctx, "faces": faces, "verts": verts, "leaf": case["leaf"],
                "rays": scenes.camera_rays_torch(_camera(seed), case["width"], case["height"], DEV)}
    if kind == "instances":
        grid, assets = case["grid"], 16
        meshes = [vt.Mesh(ctx, *_asset(case["subdivisions"], a)) for a in range(assets)]
        rng = np.random.default_rng(seed)
        n = grid * grid
        k = np.arange(n)
        angle, size = rng.uniform(0, 2 * np.pi, n), 0.4 * rng.uniform(0.8, 1.2, n)
        mirror = np.where(rng.random(n) < 0.1, -1.0, 1.0)
        t = np.zeros((n, 3, 4))
        t[:, 0, 0], t[:, 0, 2] = np.cos(angle) * size * mirror, np.sin(angle) * size
        t[:, 1, 1] = size
        t[:, 2, 0], t[:, 2, 2] = -np.sin(angle) * size * mirror, np.cos(angle) * size
        t[:, 0, 3], t[:, 1, 3], t[:, 2, 3] = k // grid - (grid - 1) / 2, 0.45, k % grid - (grid - 1) / 2
        tlas = vt.Tlas(ctx, meshes, instances_array(t, rng.integers(0, assets, n)))
        rays = _rays(case, seed)
        rays[:, 0:3] = (rays[:, 0:3] - 0.5) * torch.tensor([grid, 1.0, grid], device=DEV) + torch.tensor([0.0, 0.5, 0.0], device=DEV)
        return {"kind": kind, "tlas": tlas, "rays": rays, "query": case["query"]}
    if kind == "cache":
        return _prepare_cache(ctx, case, seed)
    return _prepare_render(ctx, case, seed)


def _prepare_render(ctx, case, seed):
    light = None
    if case["scene"] == "cornell" and case["path"] != "restir":
        faces, verts, mats, light, camera = scenes.cornell_box(seed=seed)
    elif case["scene"] == "cornell":
        faces, verts, mats, camera = scenes.cornell_emitters(seed=seed)
    else:
        faces, verts, mats, camera = _grid_scene(case["scene"])
        rng = np.random.default_rng(seed)
        mats = [dict(m, albedo=tuple(float(x) for x in rng.random(3))) if m["type"] != 3 else m for m in mats]
        # A new viewpoint over the same grid.
        a, (x, y, z) = 2 * math.pi * rng.random(), camera["pos"]
        camera = dict(camera, pos=(math.cos(a) * x + math.sin(a) * z, y, -math.sin(a) * x + math.cos(a) * z))
    mesh = vt.Mesh(ctx, faces, verts)
    scene = vt.Scene(ctx, mesh, mats, light, _spectral_tables() if case["spectral"] else None)
    mode = 0 if case["path"] == "restir" else 1
    params = vt.make_params(camera, case["width"], case["height"], case["depth"], 1, case["spectral"], mode,
                            sampler=case["sampler"], di_candidates=16 if mode == 0 else 0)
    return {"kind": "render", "scene": scene, "mesh": mesh, "params": params, "spp": case["spp"], "path": case["path"]}


def _cache_arrays(case, seed):
    rng = np.random.default_rng(seed)
    n = case["records"]
    x = np.zeros((n, nrc.INPUT_FLOATS), np.float32)
    # Path vertices lie on surfaces: points on the walls of the unit box, a few strays inside.
    p = rng.uniform(-0.95, 0.95, (n, 3))
    wall = rng.integers(0, 8, n)
    for a in range(3):
        p[wall == 2 * a, a], p[wall == 2 * a + 1, a] = -0.95, 0.95
    x[:, 0:3] = p
    x[:, 3] = np.where(rng.random(n) < 0.7, 1.0, rng.random(n))
    x[:, 4:13] = rng.random((n, 9))
    y = rng.gamma(0.7, 1.0, (n, nrc.OUTPUTS)).astype(np.float32)
    mlp = np.zeros(nrc.MLP_PARAMS, np.float32)
    mlp[:5 * 4096] = rng.uniform(-0.25, 0.25, 5 * 4096)
    mlp[5 * 4096:5 * 4096 + 256] = rng.uniform(-0.25, 0.25, 256)
    table = rng.uniform(-1, 1, case["levels"] * 2 ** case["log2_table"] * 2).astype(np.float32)
    return x, y, mlp, table


def _prepare_cache(ctx, case, seed):
    x, y, mlp, table = _cache_arrays(case, seed)
    cache = nrc.RadianceCache(ctx, [-1, -1, -1], [1, 1, 1], levels=case["levels"], log2_table=case["log2_table"],
                              base_resolution=16, max_resolution=512, spectral=int(case["spectral"]))
    cache.set_params(mlp, table)
    frame = _prepare_render(ctx, dict(case, scene="cornell", path="wavefront", sampler=0), seed)
    return dict(frame, kind="cache", cache=cache, x=x, y=y)


# ---- one pass ---------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "trace":
        if state["query"] == "any":
            return {"occluded": state["mesh"].occluded(state["rays"])}
        hits = state["mesh"].closest(state["rays"])
        return {"t_b1_b2": hits[:, :3], "face": hits[:, 3].view(torch.int32)}
    if kind == "host":
        if state["query"] == "any":
            return {"occluded": state["mesh"].occluded(state["rays"])}
        hits = state["mesh"].closest(state["rays"])
        return {"t": hits["t"], "b1": hits["b1"], "b2": hits["b2"], "face": hits["prim"]}
    if kind == "rebuild":
        mesh = vt.Mesh(state["ctx"], state["faces"], state["verts"], leaf_size=state["leaf"])
        hits = mesh.closest(state["rays"])
        info = mesh.info()
        return {"t_b1_b2": hits[:, :3], "face": hits[:, 3].view(torch.int32), "nodes": int(info.wide_nodes),
                "depth": int(info.depth), "sah": float(info.sah_cost)}
    if kind == "instances":
        if state["query"] == "any":
            return {"occluded": state["tlas"].occluded(state["rays"])}
        hits, instance = state["tlas"].closest(state["rays"])
        return {"t_b1_b2": hits[:, :3], "face": hits[:, 3].view(torch.int32), "instance": instance}
    if kind == "cache":
        mlp, grid, loss = state["cache"].gradients(state["x"], state["y"])
        state["scene"].reset()
        state["cache"].render(state["scene"], state["params"], state["spp"], train=False)
        image, _ = state["scene"].readback()
        return {"image": image, "mlp_grad": mlp, "grid_grad": grid, "loss": loss}
    scene = state["scene"]
    scene.reset()
    render = scene.render_wavefront if state["path"] == "wavefront" else scene.render
    render(state["params"], state["spp"])
    image, samples = scene.readback()
    return {"image": image, "samples": samples}


# ---- what a pass cannot do without --------------------------------------------------------------------------
def _ray_flops(faces):
    """A ray's least traversal: one 4-wide node per level (24 operations a child) and two triangle tests."""
    return 4 * 24 * max(1.0, math.log(max(faces, 4), 4)) + 2 * 60


def work(case):
    kind = case["kind"]
    if kind in ("trace", "host"):
        # Rays in, hits out, the triangles once.
        out = 1 if case["query"] == "any" else 16
        return {"bytes": case["rays"] * (32 + out) + 48 * case["faces"], "flops": case["rays"] * _ray_flops(case["faces"])}
    if kind == "rebuild":
        rays = case["width"] * case["height"]
        # Faces and vertices in; triangles and about a 4-wide node per three faces out; then the frame.
        return {"bytes": case["faces"] * (16 + 96 + 48 + 128 // 3) + 48 * rays,
                "flops": rays * _ray_flops(case["faces"]) + 200 * case["faces"]}
    if kind == "instances":
        faces = 20 * 4 ** case["subdivisions"]
        out = 1 if case["query"] == "any" else 20
        return {"bytes": case["rays"] * (32 + out) + 16 * 48 * faces + 128 * case["grid"] ** 2,
                "flops": case["rays"] * (_ray_flops(faces) + _ray_flops(case["grid"] ** 2))}
    if kind == "cache":
        n = case["records"]
        macs = 5 * 64 * 64 + 64 * 4
        grid = case["levels"] * 2 ** case["log2_table"] * 2 * 4
        paths = case["width"] * case["height"] * case["spp"]
        # Forward and backward (two products) of the records; two vertices and a prediction a path.
        return {"bytes": n * (64 + 16) + 2 * grid + 2 * 4 * nrc.MLP_PARAMS + 24 * case["width"] * case["height"],
                "flops": n * 2 * macs * 3 + paths * (2 * macs + 2 * (2 * _ray_flops(36) + 300))}
    paths = case["width"] * case["height"] * case["spp"]
    faces = {"cornell": 36, "lambert": 300_000, "production": 740_000}[case["scene"]]
    # About three vertices a path: a closest and a shadow ray each, and shading.
    return {"bytes": 48 * faces + 24 * case["width"] * case["height"], "flops": paths * 3 * (2 * _ray_flops(faces) + 300)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("trace", "host", "instances"):
        # fp32 hit distances and barycentrics; faces that meet a ray at the same distance are ties.
        return "exact" if case["query"] == "any" else {"rel": 1e-5, "max": 1e-3, "differ": 1e-5}
    if kind == "rebuild":
        return {"rel": 1e-5, "max": 1e-3, "differ": 1e-5}
    if kind == "cache":
        # fp16 operands, fp32 sums in any order.
        return {"rel": 2e-3, "max": 0.05, "differ": 0.0}
    # A path's fp32 contributions in another order; a path at a rounding edge goes another way.
    return {"rel": 2e-3, "max": 0.99, "differ": 0.0}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------
def _closest_64(faces, verts, rays):
    """Nearest hits by testing every triangle (Moeller and Trumbore 1997), in float64: (n, 3) t, b1, b2."""
    p = verts[:, :3].double()[faces[:, :3].long()]
    a, e1, e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    out = torch.zeros(len(rays), 3, dtype=torch.float64, device=rays.device)
    step = max(1, 12_000_000 // len(a))
    for i in range(0, len(rays), step):
        r = rays[i:i + step].double()
        o, d = r[:, None, 0:3], r[:, None, 4:7]
        q = torch.linalg.cross(d.expand(-1, len(a), 3), e2.expand(len(r), -1, 3))
        det = (e1 * q).sum(2)
        s = o - a
        u = (s * q).sum(2) / det
        w = torch.linalg.cross(s, e1.expand(len(r), -1, 3))
        v = (d * w).sum(2) / det
        t = (e2 * w).sum(2) / det
        ok = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= r[:, None, 3]) & (t < r[:, None, 7])
        best, at = torch.where(ok, t, torch.inf).min(1)
        found = torch.isfinite(best)
        row = torch.arange(len(r), device=rays.device)
        out[i:i + step] = torch.where(found[:, None], torch.stack([best, u[row, at], v[row, at]], 1), 0.0)
    return out


def _cache_64(case, seed):
    """The cache's definition in float64: encoding, MLP, relative L2 loss and its gradients (the frame
    has no such value)."""
    x, y, mlp, table = (torch.from_numpy(v).to(DEV) for v in _cache_arrays(case, seed))
    levels, entries = case["levels"], 2 ** case["log2_table"]
    mlp, table = mlp.double().requires_grad_(True), table.double().view(levels, entries, 2).requires_grad_(True)
    extent = float(np.float32(2.0) * np.float32(1.02))
    q = ((x[:, :3].double() + 0.5 * extent) / extent).clamp(0, 1)
    growth = math.exp((math.log(512) - math.log(16)) / (levels - 1))
    blob = lambda s: torch.exp(-8.0 * (s.double()[:, None] - (torch.arange(4, device=DEV) + 0.5) / 4) ** 2)  # noqa: E731
    feats = []
    for level in range(levels):
        res = int(math.floor(16 * growth ** level + 1e-6))
        c = (q * res).long().clamp(max=res - 1)
        f = q * res - c
        total = 0.0
        for k in range(8):
            bit = [k & 1, (k >> 1) & 1, k >> 2]
            g = [c[:, a] + bit[a] for a in range(3)]
            if (res + 1) ** 3 <= entries:
                idx = g[0] + (res + 1) * (g[1] + (res + 1) * g[2])
            else:
                idx = (g[0] ^ (g[1] * 2654435761) ^ (g[2] * 805459861)) & (entries - 1)
            w = math.prod([f[:, a] if bit[a] else 1 - f[:, a] for a in range(3)])
            total = total + w[:, None] * table[level][idx]
        feats.append(total)
    feats += [torch.zeros(len(x), 32 - 2 * levels, dtype=torch.float64, device=DEV)]
    feats += [blob(x[:, 4 + a]) for a in range(4)] + [blob(1 - torch.exp(-x[:, 3].double()))]
    feats += [x[:, 8:12].double(), blob(x[:, 12]), torch.sin(2 * math.pi * q), torch.ones(len(x), 1, dtype=torch.float64, device=DEV)]
    h = torch.cat(feats, 1)
    for layer in range(5):
        h = torch.relu(h @ mlp[layer * 4096:(layer + 1) * 4096].view(64, 64).T)
    pred = h @ mlp[5 * 4096:].view(16, 64)[:4].T
    lum = torch.tensor([0.25] * 4 if case["spectral"] else [0.2126, 0.7152, 0.0722, 0.0], dtype=torch.float64, device=DEV)
    loss = (((pred - y.double()) ** 2).sum(1) / ((pred.detach() @ lum) ** 2 + 0.01)).sum()
    loss.backward()
    # A grid entry's gradient comes from a few records, and a ReLU near zero that fp16 operands turn
    # changes such a record's share whole: 64 bits say nothing about it at this precision.
    return {"image": None, "mlp_grad": mlp.grad, "grid_grad": None, "loss": float(loss.detach())}


def exact(case, seed):
    if case["kind"] == "cache":
        return _cache_64(case, seed)
    if case["kind"] == "trace" and case["query"] == "closest" and case["faces"] * case["rays"] <= 1 << 30:
        faces, verts = _soup(case["faces"], seed)
        return {"t_b1_b2": _closest_64(faces, verts, _rays(case, seed)), "face": None}
    return None
