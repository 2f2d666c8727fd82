"""Rays from far outside their scene, aimed at triangles' edges and corners,
over the grid nodes: every hit of the linear loop is found.  Rounding moves
such a hit by about 2^-23 of the origin's distance, against boxes padded by
2^-18 of the scene's largest coordinate, so beyond some 60 scene sizes the box
tests need a margin of their own (csrc/grid.cuh: kGridSlack).  The triangles
face the rays within 75 degrees, where that bound on the triangle test holds;
results are equal bit for bit."""
import numpy as np
import pytest

from igx_raytracing_gb300 import scenes
from igx_raytracing_gb300._capi import HIT_DTYPE
from oracle import pyoracle

pytestmark = pytest.mark.gpu

SPHERE = np.array([[0.5, 0.5, 0.5, 0.02]], np.float32)


def _unit(v):
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _scene_and_rays(distance, n=30000, seed=8201):
    rng = np.random.default_rng(seed)
    tris = scenes.random_triangles(2000, seed)
    normal = _unit(np.stack([*rng.uniform(-0.7, 0.7, (2, 2000)), np.ones(2000)], 1))  # within 45 degrees of z
    a = _unit(np.cross(normal, rng.normal(size=(2000, 3))))
    b = np.cross(normal, a)
    c = rng.uniform(0, 1, (2000, 3))
    for k, f in enumerate(("p0", "p1", "p2")):
        w = 2 * np.pi * k / 3
        tris[f] = c + 0.01 * (np.cos(w) * a + np.sin(w) * b)
    d = _unit(np.stack([*rng.uniform(-0.4, 0.4, (2, n)), rng.choice([-1.0, 1.0], n)], 1))  # within 30 degrees of z
    k = rng.integers(0, 2000, n)
    w = np.where(rng.random(n) < 0.3, 0.0, rng.uniform(0, 1, n))[:, None]  # corners, else edges
    target = tris["p0"][k].astype(np.float64) * (1 - w) + tris["p1"][k].astype(np.float64) * w
    # not near the sphere, whose own test cancels at such distances
    keep = np.linalg.norm(np.cross(SPHERE[0, :3] - target, d), axis=1) > 0.1
    target, d = target[keep], d[keep]
    org = (target - distance * d).astype(np.float32)
    rays = scenes.incoherent_rays(len(org), 1)
    rays["org"], rays["dir"] = org, _unit(target - org.astype(np.float64))
    return tris, rays


def _same(got, want, ok):
    for f in ("prim", "t", "u", "v"):
        a, b = got[f][ok].view(np.uint32), want[f][ok].view(np.uint32)
        assert np.array_equal(a, b), f"{f} differs on {(a != b).sum()} of {ok.sum()} rays"


@pytest.mark.parametrize("distance", [10.0, 100.0, 1000.0, 10000.0])
def test_edges_from_far_away(ctx, distance):
    import torch

    tris, rays = _scene_and_rays(distance)
    want, flags = pyoracle.trace_geometry(tris, rays)
    ok = flags == 0
    assert (want["prim"][ok] != 0xFFFFFFFF).mean() > 0.3
    scene = ctx.create_scene(tris)
    _same(scene.trace_geometry(rays), want, ok)
    occ, flags = pyoracle.trace_occlusion(tris, rays)
    assert np.array_equal(scene.trace_occlusion(rays)[flags == 0], occ[flags == 0])
    d_rays = torch.from_numpy(rays.view(np.float32).reshape(-1, 8).copy()).cuda()
    out = torch.empty(len(rays), 4, device="cuda")
    ctx.trace_batch([(scene, d_rays, None, out, 0)])
    torch.cuda.synchronize()
    _same(out.cpu().numpy().view(HIT_DTYPE).reshape(-1), want, ok)
    scene.close()
    mixed = ctx.create_scene_mixed(tris, SPHERE)
    want, flags = pyoracle.trace_geometry_mixed(rays, None, tris=tris, spheres=SPHERE)
    _same(mixed.trace_geometry(rays), want, flags == 0)
    mixed.close()
