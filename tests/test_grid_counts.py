"""The fetch counts that the benchmark's bytes are made of, over the grid
nodes: known for a one-leaf scene and for rays that miss the scene's box, and
about those of the exact BVH4 nodes elsewhere."""
import math

import numpy as np
import pytest

import bench
from igx_raytracing_gb300 import IgxrtError, scenes
from test_exact_nodes import limited

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
def test_grid_fetch_counts(ctx, mode):
    three = scenes.random_triangles(3, 8601, mu=math.log(0.3))
    rays = scenes.incoherent_rays(500, 8602)
    rays["org"][::2] += 50.0
    rays["dir"][::2] = np.abs(rays["dir"][::2]) + 0.1  # away from the scene
    one = ctx.create_scene_gpu(three)  # at most max_leaf_size objects: one leaf
    assert bench.traced_nodes(one, 0) == bench.GRID and bench.traced_nodes(one, 2) == 2
    nf, pf = bench.count_fetches(ctx, one, rays, None, mode, bench.GRID)
    assert (nf == 1).all() and (pf[::2] == 0).all() and set(np.unique(pf)) <= {0, 3} and pf.max() == 3
    one.close()
    scene = ctx.create_scene(scenes.random_triangles(20000, 8603, mu=math.log(0.02)))
    rays = scenes.incoherent_rays(4000, 8604)
    gn, gp = bench.count_fetches(ctx, scene, rays, None, mode, bench.GRID)
    en, ep = bench.count_fetches(ctx, scene, rays, None, mode, 1)
    for g, e in ((gn, en), (gp, ep)):  # boxes a step larger, another order among equals
        assert 0.9 < g.mean() / e.mean() < 1.2
    scene.close()


def test_counts_need_a_scene_on_the_grid():
    c = limited(0)
    scene = c.create_scene(scenes.random_triangles(100, 8605))
    assert bench.traced_nodes(scene, 0) == 0
    with pytest.raises(IgxrtError):
        bench.count_fetches(c, scene, scenes.incoherent_rays(10, 1), None, 0, bench.GRID)
    scene.close()
    c.close()
