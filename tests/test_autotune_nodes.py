"""The autotuner where BVH2 and BVH4 name the same launch (over grid nodes):
one of the two is a candidate, and cached entries timed on other nodes are not
served."""
import math
import os

import pytest

from igx_raytracing_gb300 import scenes

pytestmark = pytest.mark.gpu


def _item(ctx):
    import torch

    scene = ctx.create_scene(scenes.random_triangles(20000, 8301, mu=math.log(0.02)))
    rays = torch.from_numpy(scenes.incoherent_rays(20000, 8302).view("f4").reshape(-1, 8).copy()).cuda()
    return scene, rays, None, torch.empty(len(rays), 4, device="cuda"), 0


@pytest.mark.parametrize("plain", [False, True])
@pytest.mark.parametrize("start", [0, 1])
def test_one_candidate_for_both_names(ctx, start, plain):
    item = _item(ctx)
    saved = ctx.launch_params
    try:
        ctx.set_launch_params(layout=start)
        for _ in range(3):  # not by the noise of two equal launches
            p, _ = ctx.autotune([item], reps=1, layouts=[0, 1], plain=plain)
            assert p["layout"] == start
    finally:
        ctx.set_launch_params(**saved)
    item[0].close()


def test_entries_of_other_nodes_are_not_served(ctx, tmp_path):
    import torch

    item = _item(ctx)
    cache = os.path.join(tmp_path, "tune.txt")
    name = torch.cuda.get_device_name(0)
    old = f"{name}|unit-test\t64 8 256 2 1 16 32\t0.0001\n"
    with open(cache, "w") as f:
        f.write(old)
    p, ms = ctx.autotune([item], reps=1, cache_path=cache, class_key="unit-test")
    assert ms > 0.0002
    text = open(cache).read()
    assert text.startswith(old) and len(text.splitlines()) == 2
    assert ctx.autotune([item], reps=1, cache_path=cache, class_key="unit-test") == (p, pytest.approx(ms, abs=1e-3))
    item[0].close()
