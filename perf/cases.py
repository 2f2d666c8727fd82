"""The ray-query work that a program built on this engine has it do.

Each case is one pass through the public Python API (Context, Scene, Batch,
Server): the small queries of a picking or probe call, the sphere frame, the
incoherent and occlusion batches, many scenes in one launch, a burst of served
requests, the G-buffer and shadow passes, scenes of all four primitive types,
and the frames whose geometry moves (refit) or changes (GPU build).  Scene and
ray distributions are those of igx_raytracing_gb300/scenes.py, made on the GPU
from a seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import igx_raytracing_gb300 as igx
from igx_raytracing_gb300._capi import CAMERA_DTYPE, CUBE_DTYPE

NO_HIT = float(np.float32(3.4028235e38))
LIGHT = (3.0, 3.0, 3.0)
EYES = {"heightfield": ((0.5, -1.0, 0.5), (0.5, 0.5, 0.0), (0.0, 0.0, 1.0)),
        "sphere": ((0.0, -3.0, 0.0), (0.0, 0.0, 0.0), (0.0, 0.0, 1.0)),
        "random": ((0.5, 0.5, -1.5), (0.5, 0.5, 0.5), (0.0, 1.0, 0.0))}


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # the smallest calls: one probe of 1,000 rays on device arrays (the
        # smallest served request's size), where launch and latency count
        {"name": "probe_1k", "kind": "trace", "scene": "heightfield", "tris": 4096, "rays": 1000,
         "camera": False, "mode": 0, "prev": False, "layout": 0},
        # the small configuration: 256x256 pinhole primaries on 4,096 triangles,
        # host arrays in and out
        {"name": "host_256", "kind": "host", "scene": "heightfield", "tris": 4096, "width": 256,
         "height": 256, "layout": 0},
        # the frame of the default benchmark: 1080p primaries, one bounce and
        # one shadow ray per hit on the 1,048,576-triangle sphere
        {"name": "step_1080p", "kind": "step", "scene": "sphere", "tris": 1048576, "width": 1920,
         "height": 1080, "layout": 0},
        # the largest batch: 4M incoherent rays over 2M random triangles
        {"name": "incoherent_4m", "kind": "trace", "scene": "random", "tris": 2097152, "rays": 4194304,
         "camera": False, "mode": 0, "prev": False, "layout": 0},
        # short any-hit rays with an excluded object (ambient occlusion), an
        # odd count, the 4-wide layout an autotuner picks for any-hit launches
        {"name": "occlusion_1m", "kind": "trace", "scene": "random", "tris": 262147, "rays": 999983,
         "camera": False, "mode": 1, "prev": True, "layout": 1},
        # many scenes of uneven size in one captured launch
        {"name": "batch_24", "kind": "batch", "scenes": 24, "max_tris": 262144, "max_rays": 524288,
         "layout": 0},
        # a burst of requests to the serving loop, host arrays, both query modes
        {"name": "serve_16", "kind": "serve", "scenes": 6, "max_tris": 262144, "requests": 16,
         "max_rays": 262144, "layout": 0},
        # the raygen pass at 1080p
        {"name": "gbuffer_1080p", "kind": "gbuffer", "scene": "sphere", "tris": 1048576, "width": 1920,
         "height": 1080, "layout": 0},
        # the shadow pass at 1080p with the reference's two samples
        {"name": "shadow_1080p", "kind": "shadow", "scene": "sphere", "tris": 1048576, "width": 1920,
         "height": 1080, "samples": 2, "layout": 0},
        # all four primitive types in one scene
        {"name": "mixed_1m", "kind": "mixed", "tris": 262144, "spheres": 16384, "cubes": 16384,
         "planes": 4, "rays": 1048576, "layout": 0},
        # a frame of moving geometry: refit from new positions, then primaries
        {"name": "refit_frame", "kind": "refit", "scene": "sphere", "tris": 1048576, "width": 1920,
         "height": 1080, "layout": 0},
        # a frame of changing geometry: tree built on the GPU, then its rays
        {"name": "build_frame", "kind": "build", "scene": "random", "tris": 300001, "rays": 524287,
         "layout": 0},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def image():
        w = log_int(61, 1920)
        return w, max(1, min(1080, int(w * rng.uniform(0.5, 0.7))))

    layout = rng.choice([0, 0, 0, 0, 0, 1, 1, 2])
    kind = rng.choice(["trace", "trace", "trace", "host", "step", "batch", "serve", "gbuffer", "shadow",
                       "mixed", "refit", "build"])
    scene = rng.choice(["sphere", "random"])
    if kind == "trace":
        return {"kind": kind, "scene": rng.choice(["heightfield", "sphere", "random"]),
                "tris": log_int(2000, 1500000), "rays": log_int(1000, 4000000), "camera": rng.random() < 0.3,
                "mode": rng.choice([0, 0, 1]), "prev": rng.random() < 0.5, "layout": layout}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(3, 24), "max_tris": log_int(8192, 262144),
                "max_rays": log_int(16384, 524288), "layout": layout}
    if kind == "serve":
        return {"kind": kind, "scenes": rng.randint(2, 6), "max_tris": log_int(16384, 262144),
                "requests": rng.randint(4, 16), "max_rays": log_int(4096, 262144), "layout": layout}
    if kind == "mixed":
        return {"kind": kind, "tris": log_int(5000, 262144), "spheres": log_int(500, 16384),
                "cubes": log_int(500, 16384), "planes": rng.randint(0, 4), "rays": log_int(20000, 1048576),
                "layout": layout}
    if kind == "build":  # a GPU-built tree has the 2- and 4-wide layouts
        return {"kind": kind, "scene": scene, "tris": log_int(5000, 1000000), "rays": log_int(10000, 1000000),
                "layout": min(layout, 1)}
    w, h = image()
    case = {"kind": kind, "scene": scene, "tris": log_int(5000, 1048576), "width": w, "height": h,
            "layout": layout}
    if kind == "shadow":
        case["samples"] = rng.choice([1, 2, 4])
    return case


# ---------------------------------------------------------------------------
# Scenes and rays, made on the GPU from a generator
# ---------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _unit(v):
    return v / torch.linalg.vector_norm(v, dim=-1, keepdim=True)


def _triangles(v0, v1, v2, normals=None):
    """(N, 12) float32 in the igxrt_triangle layout."""
    t = torch.zeros(len(v0), 12, device="cuda")
    t[:, 0:3], t[:, 4:7], t[:, 8:11] = v0.float(), v1.float(), v2.float()
    if normals is not None:
        t.view(torch.int32)[:, 3::4] = normals
    return t


def _quads(v00, v10, v11, v01, normals=None):
    tri = [torch.stack(p, 1).reshape(-1, 3) for p in ((v00, v00), (v10, v11), (v11, v01))]
    return _triangles(*tri, normals)


def _heightfield(tris, g):
    nx = max(1, round(math.sqrt(tris)))
    ny = max(1, tris // (2 * nx))
    ys, xs = torch.meshgrid(torch.linspace(0, 1, ny + 1, dtype=torch.float64, device="cuda"),
                            torch.linspace(0, 1, nx + 1, dtype=torch.float64, device="cuda"), indexing="ij")
    z = torch.zeros_like(xs)
    for f, a, p in zip(*(_uniform(g, 3, 4).tolist())):
        a, p, f = 2 * math.pi * a, 2 * math.pi * p, 1 + 7 * f
        z += 0.05 * torch.sin(2 * math.pi * f * (xs * math.cos(a) + ys * math.sin(a)) + p)
    v = torch.stack([xs, ys, z], -1)
    return _quads(*(q.reshape(-1, 3) for q in (v[:-1, :-1], v[:-1, 1:], v[1:, 1:], v[1:, :-1])))


def _sphere(tris, g):
    """The displaced lat-long sphere, with vertex normals as two half words."""
    nlat = max(4, round(math.sqrt(tris / 4)))
    nlon = max(4, tris // (2 * nlat))
    th = torch.linspace(0, math.pi, nlat + 1, dtype=torch.float64, device="cuda")[:, None]
    ph = torch.arange(nlon, dtype=torch.float64, device="cuda")[None] * (2 * math.pi / nlon)
    r = 1 + 0.02 * _normal(g, nlat + 1, nlon)
    v = torch.stack([r * torch.sin(th) * torch.cos(ph), r * torch.sin(th) * torch.sin(ph),
                     r * torch.cos(th).expand(-1, nlon)], -1)
    v = torch.cat([v, v[:, :1]], 1)
    half = (0.7 * _uniform(g, 2 * nlat * nlon, 3, 2)).half().view(torch.int32).squeeze(-1)
    return _quads(*(q.reshape(-1, 3) for q in (v[:-1, :-1], v[:-1, 1:], v[1:, 1:], v[1:, :-1])), half)


def _random(tris, g):
    """Equilateral triangles in the unit cube, edges log-normal around 0.005."""
    c = _uniform(g, tris, 3)
    edge = torch.exp(math.log(0.005) + 0.7 * _normal(g, tris, 1))
    a = _unit(_normal(g, tris, 3))
    b = _unit(torch.linalg.cross(a, _normal(g, tris, 3)))
    s3 = math.sqrt(3.0)
    return _triangles(c + edge * a / s3, c + edge * (b / 2 - a / (2 * s3)), c - edge * (b / 2 + a / (2 * s3)))


SCENES = {"heightfield": _heightfield, "sphere": _sphere, "random": _random}


def _host(t):
    return t.cpu().numpy().view(igx.TRIANGLE_DTYPE).reshape(-1)


def _pinhole(scene, width, height):
    """Eye and the corners p0 (top left), p1 (top right), p2 (bottom left)."""
    eye, target, up = (np.array(v, np.float64) for v in EYES[scene])
    fwd = (target - eye) / np.linalg.norm(target - eye)
    right = np.cross(fwd, up)
    right /= np.linalg.norm(right)
    upv = np.cross(right, fwd)
    h = math.tan(math.radians(30.0))
    a = h * width / height
    return eye, eye + fwd - a * right + h * upv, eye + fwd + a * right + h * upv, eye + fwd - a * right - h * upv


def _rays(org, dirs, tmax=NO_HIT):
    r = torch.zeros(len(dirs), 8, device="cuda")
    r[:, 0:3], r[:, 4:7] = org.float(), dirs.float()
    r[:, 7] = tmax
    return r


def _camera_rays(scene, width, height, g, count=None):
    """Primaries with one jitter per image, rows from the bottom."""
    eye, p0, p1, p2 = (torch.tensor(v, device="cuda") for v in _pinhole(scene, width, height))
    jitter = _uniform(g, 2)
    ys, xs = torch.meshgrid(torch.arange(height, device="cuda"), torch.arange(width, device="cuda"), indexing="ij")
    cx = (xs.reshape(-1, 1)[:count] + jitter[0]) / width
    cy = 1 - (ys.reshape(-1, 1)[:count] + jitter[1]) / height
    return _rays(eye, _unit(p0 + cx * (p1 - p0) + cy * (p2 - p0) - eye))


def _camera(scene, width, height, g):
    c = np.zeros(1, CAMERA_DTYPE)
    c["eye"], c["p0"], c["p1"], c["p2"] = _pinhole(scene, width, height)
    c["width"], c["height"] = width, height
    c["jitter_x"], c["jitter_y"] = _uniform(g, 2).tolist()
    return c


def _incoherent(n, g, tmax=NO_HIT):
    return _rays(_uniform(g, n, 3), _unit(_normal(g, n, 3)), tmax)


def _secondary(tris, primary, hits, g, count=None):
    """Per primary hit: a cosine-weighted bounce and a shadow ray to the light,
    with the hit triangle excluded; also the pixels that hit.  With `count`,
    that many of the hits in pixel order (evenly spread)."""
    prim = hits.view(torch.int32)[:, 3]
    hit = torch.nonzero(prim != -1)[:, 0]
    if count is not None:
        hit = hit[torch.arange(count, device="cuda") * len(hit) // count]
    prim, ray, t = prim[hit], primary[hit].double(), hits[hit][:, 0:1].double()
    p = ray[:, 0:3] + t * ray[:, 4:7]
    v = tris[prim.long()].double()
    n = _unit(torch.linalg.cross(v[:, 4:7] - v[:, 0:3], v[:, 8:11] - v[:, 0:3]))
    n = torch.where((n * ray[:, 4:7]).sum(1, keepdim=True) > 0, -n, n)
    bounce = _rays(p, _unit(n + 0.999 * _unit(_normal(g, len(p), 3))))
    to_light = torch.tensor(LIGHT, dtype=torch.float64, device="cuda") - p
    dist = torch.linalg.vector_norm(to_light, dim=1, keepdim=True)
    return bounce, _rays(p, to_light / dist, dist[:, 0].float()), prim.contiguous(), hit


def _closest_out(n):
    """A closest-hit output and its parts: t, (u, v) and the object word."""
    out = torch.empty(n, 4, device="cuda")
    return out, {"t": out[:, 0], "uv": out[:, 1:3], "prim": out.view(torch.int32)[:, 3]}


def _log_sizes(lo, hi, n):
    """n sizes, log-uniform over [lo, hi] in mixed order, the largest among them."""
    x = math.log(lo) + _uniform(_generator(n), n) * (math.log(hi) - math.log(lo))
    s = [int(v) for v in torch.exp(x).tolist()]
    s[0] = int(hi)
    return s


# ---------------------------------------------------------------------------
# prepare, run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    g = _generator(seed)
    ctx = igx.Context(0)
    ctx.set_launch_params(layout=case["layout"])
    s = {"kind": case["kind"], "ctx": ctx}
    return globals()["_prepare_" + case["kind"]](case, g, s)


def run(s):
    return globals()["_run_" + s["kind"]](s)


def _prepare_trace(case, g, s):
    tris = SCENES[case["scene"]](case["tris"], g)
    s["scene"] = s["ctx"].create_scene(_host(tris))
    n = case["rays"]
    if case["camera"]:
        side = math.ceil(math.sqrt(n))
        rays = _camera_rays(case["scene"], side, side, g, n)
    else:
        rays = _incoherent(n, g)
    if case["mode"]:  # occlusion rays end at a light or a radius
        rays[:, 7] = (0.05 + 0.45 * _uniform(g, n)).float() * (8 if case["camera"] else 1)
    s["rays"], s["mode"] = rays, case["mode"]
    s["prev"] = (torch.randint(len(tris), (n,), generator=g, device="cuda", dtype=torch.int32)
                 if case["prev"] else None)
    if case["mode"]:
        s["out"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["parts"] = {"occluded": s["out"]}
    else:
        s["out"], s["parts"] = _closest_out(n)
    return s


def _run_trace(s):
    trace = s["ctx"].trace_any if s["mode"] else s["ctx"].trace_closest
    trace(s["scene"], s["rays"], s["prev"], out=s["out"])
    return s["parts"]


def _prepare_host(case, g, s):
    tris = SCENES[case["scene"]](case["tris"], g)
    s["scene"] = s["ctx"].create_scene(_host(tris))
    rays = _camera_rays(case["scene"], case["width"], case["height"], g)
    s["rays"] = rays.cpu().numpy().view(igx.RAY_DTYPE).reshape(-1)
    return s


def _run_host(s):
    hits = s["scene"].trace_geometry(s["rays"])
    return {"t": hits["t"], "u": hits["u"], "v": hits["v"], "prim": hits["prim"]}


def _prepare_step(case, g, s):
    ctx = s["ctx"]
    tris = SCENES[case["scene"]](case["tris"], g)
    s["scene"] = ctx.create_scene(_host(tris))
    s["primary"] = _camera_rays(case["scene"], case["width"], case["height"], g)
    s["hits"], first = _closest_out(len(s["primary"]))
    ctx.trace_closest(s["scene"], s["primary"], out=s["hits"])
    # the sphere covers 18% of the image: that many secondary rays
    count = max(1, int(0.18 * len(s["primary"])))
    s["bounce"], s["shadow"], s["prev"], _ = _secondary(tris, s["primary"], s["hits"], g, count)
    s["bounce_hits"], second = _closest_out(len(s["bounce"]))
    s["occluded"] = torch.empty(len(s["shadow"]), dtype=torch.int32, device="cuda")
    s["parts"] = {"primary": first, "bounce": second, "occluded": s["occluded"]}
    return s


def _run_step(s):
    ctx, scene = s["ctx"], s["scene"]
    ctx.trace_closest(scene, s["primary"], out=s["hits"])
    ctx.trace_closest(scene, s["bounce"], s["prev"], out=s["bounce_hits"])
    # made from the primary hits: independent of the bounce launch before it
    ctx.trace_any(scene, s["shadow"], s["prev"], out=s["occluded"], independent=True)
    return s["parts"]


def _prepare_batch(case, g, s):
    k = case["scenes"]
    s["scenes"], s["items"], s["parts"] = [], [], []
    sizes = zip(_log_sizes(1024, case["max_tris"], k), _log_sizes(4096, case["max_rays"], k)[::-1])
    for i, (tris, n) in enumerate(sizes):
        scene = s["ctx"].create_scene(_host(_random(tris, g)))
        half = n // 2  # half pinhole primaries, half incoherent
        side = max(1, math.ceil(math.sqrt(half)))
        rays = torch.cat([_camera_rays("random", side, side, g, half), _incoherent(n - half, g)])
        out, parts = _closest_out(n)
        s["scenes"].append(scene)
        s["items"].append((scene, rays, None, out, 0))
        s["parts"].append([parts["t"], parts["prim"]])
    s["batch"] = s["ctx"].create_batch(s["items"])
    return s


def _run_batch(s):
    s["batch"].launch()
    return s["parts"]


def _prepare_serve(case, g, s):
    s["server"] = igx.Server(s["ctx"], memory_cap_bytes=2 << 30)
    s["scenes"] = [s["ctx"].create_scene(_host(_random(n, g)))
                   for n in _log_sizes(10000, case["max_tris"], case["scenes"])]
    ids = [s["server"].add_scene(x) for x in s["scenes"]]
    s["requests"], s["parts"] = [], []
    for i, n in enumerate(_log_sizes(1000, case["max_rays"], case["requests"])):
        rays = _incoherent(n, g).cpu().pin_memory().numpy().view(igx.RAY_DTYPE).reshape(-1)
        mode = i % 2
        out = (torch.empty(n, dtype=torch.int32) if mode else torch.empty(n, 4)).pin_memory().numpy()
        s["requests"].append((ids[i % len(ids)], rays, None, mode, out))
        s["parts"].append([out] if mode else [out[:, 0], out[:, 1:3], out.view(np.int32)[:, 3]])
    return s


def _run_serve(s):
    server = s["server"]
    tickets = [server.submit(*q) for q in s["requests"]]
    for t in tickets:
        server.wait(t)
    return s["parts"]


def _prepare_gbuffer(case, g, s):
    w, h = case["width"], case["height"]
    s["scene"] = s["ctx"].create_scene(_host(SCENES[case["scene"]](case["tris"], g)))
    s["camera"] = _camera(case["scene"], w, h, g)
    a, b = torch.empty(h, w, 4, device="cuda"), torch.zeros(h, w, 4, device="cuda")
    s["images"] = a, b
    s["parts"] = {"dir": a[..., 0:3], "object": a.view(torch.int32)[..., 3], "uv": b[..., 0:2],
                  "normal": b.view(torch.int32)[..., 2:4]}
    return s


def _run_gbuffer(s):
    s["ctx"].trace_gbuffer(s["scene"], s["camera"], *s["images"])
    return s["parts"]


def _prepare_shadow(case, g, s):
    ctx, w, h, k = s["ctx"], case["width"], case["height"], case["samples"]
    tris = SCENES[case["scene"]](case["tris"], g)
    s["scene"] = ctx.create_scene(_host(tris))
    primary = _camera_rays(case["scene"], w, h, g)
    hits = ctx.trace_closest(s["scene"], primary)
    s["object"] = hits.view(torch.int32)[:, 3].contiguous()
    s["rays"] = torch.zeros(k * w * h, 8, device="cuda")
    for j in range(k):  # each sample toward its own point of the light
        _, shadow, _, hit = _secondary(tris, primary, hits, g)
        shadow[:, 4:7] = _unit(shadow[:, 4:7].double() + 0.02 * _normal(g, len(shadow), 3)).float()
        s["rays"][j * w * h:(j + 1) * w * h][hit] = shadow
    s["size"] = w, h, k
    s["mask"] = torch.zeros(((w + 15) // 16) * ((h + 1) // 2) * k, dtype=torch.int32, device="cuda")
    return s


def _run_shadow(s):
    return s["ctx"].trace_shadow_mask(s["scene"], s["rays"], s["object"], *s["size"], out=s["mask"])


def _prepare_mixed(case, g, s):
    c = _uniform(g, case["spheres"], 3)
    spheres = torch.cat([c, torch.exp(math.log(0.004) + 0.5 * _normal(g, case["spheres"], 1))], 1)
    lo = _uniform(g, case["cubes"], 3)
    cubes = torch.cat([lo, lo + torch.exp(math.log(0.006) + 0.5 * _normal(g, case["cubes"], 3))], 1)
    planes = [(0.0, 0.0, 1.0, 0.05), (1.0, 0.0, 0.0, 0.05), (-1.0, 0.0, 0.0, -1.05), (0.0, 1.0, 0.0, 0.05)]
    s["scene"] = s["ctx"].create_scene_mixed(
        _host(_random(case["tris"], g)), spheres.float().cpu().numpy(),
        cubes.float().cpu().numpy().view(CUBE_DTYPE).reshape(-1),
        np.array(planes[:case["planes"]], np.float32).reshape(-1, 4))
    s["rays"] = _incoherent(case["rays"], g)
    s["out"], s["parts"] = _closest_out(case["rays"])
    return s


def _run_mixed(s):
    s["ctx"].trace_closest(s["scene"], s["rays"], out=s["out"])
    return s["parts"]


def _prepare_refit(case, g, s):
    tris = SCENES[case["scene"]](case["tris"], g)
    s["scene"] = s["ctx"].create_scene(_host(tris))
    s["moved"] = tris.clone()
    amp, turn = 0.02 + 0.04 * _uniform(g, 1), 6.0 * _uniform(g, 1)
    for k in (0, 4, 8):  # a breathing deformation of every vertex
        p = tris[:, k:k + 3].double()
        s["moved"][:, k:k + 3] = (p * (1 + amp * torch.sin(3 * p[:, 2:3] + turn))).float()
    s["rays"] = _camera_rays(case["scene"], case["width"], case["height"], g)
    s["out"], s["parts"] = _closest_out(len(s["rays"]))
    return s


def _run_refit(s):
    s["scene"].refit(s["moved"])
    s["ctx"].trace_closest(s["scene"], s["rays"], out=s["out"])
    return s["parts"]


def _prepare_build(case, g, s):
    s["tris"] = SCENES[case["scene"]](case["tris"], g)
    s["rays"] = _incoherent(case["rays"], g)
    s["out"], s["parts"] = _closest_out(case["rays"])
    return s


def _run_build(s):
    # the previous frame's scene goes once this frame's is there
    s["scene"] = s["ctx"].create_scene_gpu(s["tris"])
    s["ctx"].trace_closest(s["scene"], s["rays"], out=s["out"])
    return s["parts"]


# ---------------------------------------------------------------------------
# What a pass cannot do without; exact results
# ---------------------------------------------------------------------------

def work(case):
    """Bytes: rays, results and the scene's primitives, each once.  Flops: a
    slab test (about 24) per level of a balanced binary tree and a triangle
    test (about 60) per ray."""
    kind = case["kind"]
    if kind in ("batch", "serve"):
        # log-uniform sizes: their mean is (hi - lo) / ln(hi / lo)
        mean = lambda lo, hi: (hi - lo) / math.log(hi / lo)
        tris = case["scenes"] * mean(1024 if kind == "batch" else 10000, case["max_tris"])
        n = case["scenes" if kind == "batch" else "requests"]
        rays = n * mean(4096 if kind == "batch" else 1000, case["max_rays"])
        depth = math.log2(tris / case["scenes"])
    else:
        tris = case["tris"] + case.get("spheres", 0) + case.get("cubes", 0)
        rays = case["rays"] if "rays" in case else case["width"] * case["height"]
        depth = math.log2(tris)
    per_ray = 32 + (4 if case.get("mode") else 16) + (4 if case.get("prev") else 0)
    if kind == "gbuffer":
        per_ray = 32  # no ray is read, two 16-byte texels are written
    if kind == "shadow":
        per_ray = 4 + 32 * 0.18 * case["samples"]  # about 18% of the pixels hit
    if kind == "step":
        per_ray += 0.18 * (2 * 36 + 16 + 4)
        rays_traced = 1.36 * rays
    else:
        rays_traced = rays * (0.18 * case["samples"] if kind == "shadow" else 1)
    # a refit also writes each primitive's record and boxes, a build its tree
    scene = 48 * tris * {"refit": 3, "build": 3}.get(kind, 1)
    return {"bytes": float(per_ray * rays + scene), "flops": float(rays_traced * (24 * depth + 60))}


def _exact_closest(tris, rays, prev=None):
    """Every triangle against every ray, in 64 bits (the smallest t > 0)."""
    v = tris.double()
    p0, e1, e2 = v[:, 0:3], v[:, 4:7] - v[:, 0:3], v[:, 8:11] - v[:, 0:3]
    best = torch.full((len(rays), 3), 0.0, dtype=torch.float64, device="cuda")
    best[:, 0] = NO_HIT
    cross, dot = torch.linalg.cross, lambda a, b: (a * b).sum(-1)
    for i in range(0, len(rays), 4096):
        o, d = rays[i:i + 4096, None, 0:3].double(), rays[i:i + 4096, None, 4:7].double()
        for j in range(0, len(v), 2048):
            h = cross(d, e2[None, j:j + 2048].expand(len(d), -1, -1), dim=-1)
            f = 1 / dot(e1[None, j:j + 2048], h)
            q0 = o - p0[None, j:j + 2048]
            u = f * dot(q0, h)
            q = cross(q0, e1[None, j:j + 2048].expand_as(q0), dim=-1)
            w = f * dot(d, q)
            t = f * dot(e2[None, j:j + 2048], q)
            ok = (u >= 0) & (u <= 1) & (w >= 0) & (u + w <= 1) & (t > 0)
            if prev is not None:
                ok &= prev[i:i + 4096, None] != torch.arange(j, j + h.shape[1], device="cuda")[None]
            t, k = torch.where(ok, t, math.inf).min(1)
            r = torch.arange(len(k), device="cuda")
            new = torch.stack([t, u[r, k], w[r, k]], 1)
            part = best[i:i + 4096]
            part[:] = torch.where((t < part[:, 0])[:, None], new, part)
    return best


def exact(case, seed):
    """Closest hits by testing every pair, where that takes seconds."""
    kind = case["kind"]
    rays = case["rays"] if "rays" in case else case.get("width", 0) * case.get("height", 0)
    if kind not in ("trace", "host", "build") or case.get("mode") or case["tris"] * rays > 4e9:
        return None
    g = _generator(seed)
    tris = SCENES[case["scene"]](case["tris"], g)
    if kind == "host":
        b = _exact_closest(tris, _camera_rays(case["scene"], case["width"], case["height"], g))
        return {"t": b[:, 0], "u": b[:, 1], "v": b[:, 2], "prim": None}
    if kind == "trace" and case["camera"]:
        side = math.ceil(math.sqrt(rays))
        r = _camera_rays(case["scene"], side, side, g, rays)
    else:
        r = _incoherent(rays, g)
    prev = None
    if case.get("prev"):
        prev = torch.randint(len(tris), (rays,), generator=g, device="cuda", dtype=torch.int32)
    b = _exact_closest(tris, r, prev)
    return {"t": b[:, 0], "uv": b[:, 1:3], "prim": None}
