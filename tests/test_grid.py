"""The grid nodes (csrc/grid.cuh: child boxes as 16-bit words on a grid over
the scene), which launches over BVH2 and BVH4 trace where the grid is fine
enough: hits against the brute-force oracle, bit for bit, where the
quantization and its rule could go wrong: nodes with absent slots, scenes far
from the origin, flat or at the ends of the float range, detail below the
grid's steps, directions that leave the range of the folded arithmetic, rays
along the grid's faces, and refits that make the grid unusable and usable
again under a captured batch."""
import math

import numpy as np
import pytest

from igx_raytracing_gb300 import scenes
from igx_raytracing_gb300._capi import HIT_DTYPE
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _check(scene, tris, rays, prev=None, what=""):
    hits = scene.trace_geometry(rays, prev)
    expect, flags = pyoracle.trace_geometry(tris, rays, prev)
    ok = flags == 0  # NaN-t rays: the linear loop's answer depends on index order alone
    assert ok.mean() > 0.5
    for f in ("prim", "t", "u", "v"):
        a, b = hits[f][ok].view(np.uint32), expect[f][ok].view(np.uint32)
        assert np.array_equal(a, b), f"{what}: {f} differs on {(a != b).sum()} of {ok.sum()} rays"
    occ = scene.trace_occlusion(rays, prev)
    want, flags = pyoracle.trace_occlusion(tris, rays, prev)
    ok = flags == 0
    assert np.array_equal(occ[ok], want[ok]), what


def _rays(n, seed, centre=(0.5, 0.5, 0.5), size=1.0):
    rays = scenes.incoherent_rays(n, seed)
    rays["org"] = ((rays["org"].astype(np.float64) - 0.5) * size + centre).astype(np.float32)
    return rays


def _moved(tris, scale=1.0, shift=(0.0, 0.0, 0.0)):
    out = tris.copy()
    for f in ("p0", "p1", "p2"):
        out[f] = (tris[f].astype(np.float64) * scale + shift).astype(np.float32)
    return out


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 9, 17, 33, 130, 1027])
def test_small_trees(ctx, n, layout):
    tris = scenes.random_triangles(n, 7100 + n, mu=math.log(0.2))
    saved = ctx.launch_params
    try:
        ctx.set_launch_params(layout=layout)
        scene = ctx.create_scene(tris)
        rays = _rays(777, 7200 + n)
        rays["dir"][:300] = tris["p1"][np.arange(300) % n] - rays["org"][:300]  # at the vertices
        prev = np.where(np.arange(777) % 3 == 0, np.arange(777) % n, 0xFFFFFFFF).astype(np.uint32)
        _check(scene, tris, rays, prev, f"{n} triangles, layout {layout}")
        scene.close()
    finally:
        ctx.set_launch_params(**saved)


@pytest.mark.parametrize("scale,shift", [(1.0, (1000.0, -500.0, 3.0)), (1e-12, (0, 0, 0)), (1e12, (0, 0, 0)),
                                         (3e14, (0, 0, 0))])
def test_scenes_over_the_float_range(ctx, scale, shift):
    tris = _moved(scenes.random_triangles(3000, 7301, mu=math.log(0.03)), scale, shift)
    scene = ctx.create_scene(tris)
    rays = _rays(2000, 7302)
    rays["org"] = (rays["org"].astype(np.float64) * scale + shift).astype(np.float32)
    rays["dir"][::5, 1:] = 0  # axis-parallel
    _check(scene, tris, rays, what=f"scale {scale} shift {shift}")
    scene.close()


def test_flat_scene(ctx):
    tris = scenes.heightfield(40, 30, 7303)
    for f in ("p0", "p1", "p2"):
        tris[f][:, 2] = 0.25
    scene = ctx.create_scene(tris)
    rays = _rays(4000, 7304)
    rays["dir"][::4, :2] = 0
    _check(scene, tris, rays, what="flat")
    scene.close()


@pytest.mark.parametrize("magnitude", [1e-12, 1e8, 1e20, 1e27])
def test_direction_magnitudes(ctx, magnitude):
    tris = scenes.random_triangles(500, 7305, mu=math.log(0.1))
    scene = ctx.create_scene(tris)
    rays = _rays(600, 7306)
    rays["dir"][::3, 0] = 0
    rays["dir"][::7, 2] = 0
    rays["dir"] = (rays["dir"].astype(np.float64) * magnitude).astype(np.float32)
    rays["tmin"][::4] = -2.0 / magnitude
    rays["tmin"][::9] = -np.inf
    _check(scene, tris, rays, what=f"|dir| {magnitude}")
    scene.close()


def test_rays_along_the_scene_box(ctx):
    """Origins on the scene box's corners and faces, directions along its
    edges and diagonals: where near and far planes coincide."""
    tris = scenes.random_triangles(4000, 7307, mu=math.log(0.05))
    p = np.concatenate([tris[f] for f in ("p0", "p1", "p2")])
    lo, hi = p.min(0).astype(np.float64), p.max(0).astype(np.float64)
    pad = np.abs(p).max() * 2.0 ** -18
    rng = np.random.default_rng(7308)
    rays = _rays(3000, 7309)
    corner = rng.integers(0, 2, (3000, 3))
    rays["org"] = np.where(corner, hi + pad, lo - pad).astype(np.float32)
    face = rng.random((3000, 3)) < 0.5
    rays["org"] = np.where(face, rays["org"], rng.uniform(lo, hi, (3000, 3))).astype(np.float32)
    d = np.where(corner, -1.0, 1.0) * (rng.random((3000, 3)) < 0.6)
    d[np.abs(d).sum(1) == 0] = (0.0, 0.0, 1.0)
    rays["dir"] = d.astype(np.float32)
    scene = ctx.create_scene(tris)
    _check(scene, tris, rays, what="scene box")
    scene.close()


def _stadium(seed):
    """A floor of extent 2000 with half its triangles in a patch of size 0.01."""
    floor = _moved(scenes.heightfield(40, 40, seed), 2000.0, (-1000.0, -1000.0, 0.0))
    detail = _moved(scenes.random_triangles(3000, seed + 1, mu=math.log(0.05)), 0.01, (3.0, 2.0, 40.0))
    return np.concatenate([floor, detail])


def test_detail_below_the_grid_steps(ctx):
    tris = _stadium(7310)
    scene = ctx.create_scene(tris)
    rays = _rays(3000, 7312, centre=(3.005, 2.005, 40.005), size=0.03)
    rays["org"][::10] = (0.0, 0.0, 300.0)
    rays["dir"][::10] = np.float32((3.005, 2.005, -259.995))
    _check(scene, tris, rays, what="stadium")
    scene.close()


@pytest.mark.parametrize("gpu_build", [False, True])
def test_refit_moves_the_grid(ctx, gpu_build):
    """Plain launches and a captured batch over a scene whose refits blow the
    grid up (one triangle far away), bring it back and shift it."""
    import torch

    tris = scenes.random_triangles(3000, 7313, mu=math.log(0.03))
    up = lambda a: torch.from_numpy(a.view(np.float32).reshape(len(a), -1).copy()).cuda()
    scene = ctx.create_scene_gpu(up(tris)) if gpu_build else ctx.create_scene(tris)
    rays = _rays(2500, 7314)
    d_rays, out = up(rays), torch.empty(len(rays), 4, device="cuda")
    batch = ctx.create_batch([(scene, d_rays, None, out, 0)])
    far = tris.copy()
    far["p0"][7] += np.float32(3e6)
    for frame, t in enumerate([tris, far, tris, _moved(tris, 0.5, (0.2, 0.3, 0.1))]):
        scene.refit(up(t))
        _check(scene, t, rays, what=f"frame {frame}")
        batch.launch()
        torch.cuda.synchronize()
        got = out.cpu().numpy().view(HIT_DTYPE).reshape(-1)
        expect, flags = pyoracle.trace_geometry(t, rays)
        ok = flags == 0
        assert np.array_equal(got["prim"][ok], expect["prim"][ok])
        assert np.array_equal(got["t"][ok].view(np.uint32), expect["t"][ok].view(np.uint32))
    batch.close()
    scene.close()
