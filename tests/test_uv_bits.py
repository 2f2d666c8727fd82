"""u and v of sphere hits from the batches of a warp, bit for bit: the engine
and the oracle both round binary64 asin and atan once to binary32."""
import numpy as np
import pytest

from igx_raytracing_gb300 import scenes
from oracle import pyoracle
from test_refit import random_mixed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [0, 1, 2])
@pytest.mark.parametrize("memory", ["host", "device"])
def test_sphere_uv_bits(ctx, layout, memory):
    import torch

    sc = random_mixed(41, nt=300, ns=4000, nc=40, npl=1)
    rays = scenes.incoherent_rays(20000, 8401)
    want, flags = pyoracle.trace_geometry_mixed(rays, None, **sc)
    ok = flags == 0
    spheres = (want["prim"] >= 300) & (want["prim"] < 4300)
    assert (ok & spheres).sum() > 5000
    scene = ctx.create_scene_mixed(sc["tris"], sc["spheres"], sc["cubes"], sc["planes"])
    saved = ctx.launch_params
    try:
        ctx.set_launch_params(layout=layout)
        if memory == "host":
            got = scene.trace_geometry(rays)
        else:
            d_rays = torch.from_numpy(rays.view(np.float32).reshape(-1, 8).copy()).cuda()
            got = ctx.trace_closest(scene, d_rays).cpu().numpy().view(want.dtype).reshape(-1)
    finally:
        ctx.set_launch_params(**saved)
    for f in ("prim", "t", "u", "v"):
        a, b = got[f][ok].view(np.uint32), want[f][ok].view(np.uint32)
        assert np.array_equal(a, b), f"{f} differs on {(a != b).sum()} rays"
    scene.close()
