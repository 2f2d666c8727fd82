"""Sphere hits' uv in batches of a warp (csrc/trace_kernels.cu: flush_uv):
hits of scenes that are mostly spheres against the oracle's linear loop, with
ray counts around the batch size, every layout's kernel, spheres behind and
in front of triangles, cubes and planes at about the same distance, and an
excluded object.  u and v within the 2 ulp of asin and atan, the rest bit for
bit."""
import numpy as np
import pytest

from igx_raytracing_gb300 import scenes
from oracle import pyoracle
from test_refit import random_mixed

pytestmark = pytest.mark.gpu
UV_ULPS = 2


def _ulps(a, b):
    ia, ib = (x.view(np.int32).astype(np.int64) for x in (a, b))
    ia, ib = (np.where(x < 0, -(x & 0x7FFFFFFF), x) for x in (ia, ib))
    return np.abs(ia - ib)


@pytest.mark.parametrize("layout", [0, 1, 2])
@pytest.mark.parametrize("triangles", [0, 400])
def test_sphere_hits(ctx, layout, triangles):
    sc = random_mixed(31, nt=max(triangles, 1), ns=3000, nc=40 if triangles else 0, npl=1 if triangles else 0)
    rays = scenes.incoherent_rays(5000, 7801)
    total = len(sc["tris"]) + len(sc["spheres"])
    prev = np.where(np.arange(5000) % 4 == 0, np.arange(5000) % total, 0xFFFFFFFF).astype(np.uint32)
    want, flags = pyoracle.trace_geometry_mixed(rays, prev, **sc)
    ok = flags == 0
    sphere = (want["prim"] >= len(sc["tris"])) & (want["prim"] < total)
    assert (sphere & ok).sum() > 1000
    scene = ctx.create_scene_mixed(sc["tris"], sc["spheres"], sc["cubes"], sc["planes"])
    saved = ctx.launch_params
    try:
        ctx.set_launch_params(layout=layout)
        for n in (1, 2, 31, 32, 33, 64, 65, 1000, 5000):
            got = scene.trace_geometry(rays[:n], prev[:n])
            k = ok[:n]
            for f in ("prim", "t"):
                assert np.array_equal(got[f][k].view(np.uint32), want[f][:n][k].view(np.uint32)), (f, n)
            for f in ("u", "v"):
                assert _ulps(got[f][k], want[f][:n][k]).max(initial=0) <= UV_ULPS, (f, n)
    finally:
        ctx.set_launch_params(**saved)
    scene.close()
