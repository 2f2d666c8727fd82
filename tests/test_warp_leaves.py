"""Leaves tested by the whole warp (csrc/leaf.cuh): hits and occluded words
against the brute-force oracle, bit for bit, with leaves from one record to
the most a leaf holds (16), so that a phase's pairs end before, on and after
its turns of 32; with rays that stop inside the scene, an excluded object,
every number of rays around a warp, and each end of the node phase."""
import math

import numpy as np
import pytest

from igx_raytracing_gb300 import BVH, scenes
from oracle import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("phase_break", [1, 2, 32])
@pytest.mark.parametrize("leaf", [1, 2, 3, 8, 15, 16])
def test_leaf_lengths(ctx, leaf, phase_break):
    tris = scenes.random_triangles(2500, 7600 + leaf, mu=math.log(0.05))
    scene = ctx.create_scene(bvh=BVH.build(tris, max_leaf_size=leaf, tri_cost=1e-3))
    rng = np.random.default_rng(7700 + leaf)
    rays = scenes.incoherent_rays(6000, 7601)
    rays["tmax"] = rng.uniform(0.02, 0.6, 6000).astype(np.float32)
    rays["tmin"] = np.where(rng.random(6000) < 0.3, 0.05, 0.0).astype(np.float32)
    prev = np.where(rng.random(6000) < 0.5, rng.integers(0, 2500, 6000), 0xFFFFFFFF).astype(np.uint32)
    want, flags = pyoracle.trace_occlusion(tris, rays, prev)
    ok = flags == 0
    assert 0.05 < want[ok].mean() < 0.95
    closest, flags = pyoracle.trace_geometry(tris, rays, prev)
    near = flags == 0
    saved = ctx.launch_params
    try:
        ctx.set_launch_params(layout=0, phase_break=phase_break)
        for n in (1, 5, 31, 32, 33, 777, 6000):
            got = scene.trace_occlusion(rays[:n], prev[:n])
            assert np.array_equal(got[ok[:n]], want[:n][ok[:n]]), (leaf, n)
            hits = scene.trace_geometry(rays[:n], prev[:n])
            for f in ("prim", "t", "u", "v"):
                a, b = (x[f][:n][near[:n]].view(np.uint32) for x in (hits, closest))
                assert np.array_equal(a, b), (leaf, n, f)
    finally:
        ctx.set_launch_params(**saved)
    scene.close()
