"""GPU-built trees whose BVH4 is deeper than the levels the build launches over
the whole GPU (csrc/lbvh.cu: kWideLevels): the last levels come from the one
block that takes what is left.  Clusters at halving distances split off one
Morton bit at a time, and thousands of equal centroids split by their ids."""
import math

import numpy as np
import pytest

from conftest import NO_HIT, assert_hits_equal
from igx_raytracing_gb300 import scenes
from igx_raytracing_gb300._capi import LAYOUT_BVH4
from oracle import pyoracle

pytestmark = pytest.mark.gpu

WIDE_LEVELS = 20


def _deep(leaf, same):
    base = scenes.random_triangles(8, 7401, mu=math.log(0.2))
    parts = []
    for bit in range(30):  # from the far corner toward the origin, one axis' bit at a time
        k, axis = bit // 3, bit % 3
        t = base.copy()
        centre = np.zeros(3)
        centre[axis] = 0.75 * 2.0 ** -k
        for f in ("p0", "p1", "p2"):
            t[f] = ((base[f].astype(np.float64) - 0.5) * 0.02 * 2.0 ** -k + centre).astype(np.float32)
        parts.append(t)
    one = scenes.random_triangles(1, 7402, mu=math.log(0.2))
    for f in ("p0", "p1", "p2"):
        one[f] = one[f] * np.float32(1e-5)
    parts.append(np.repeat(one, same))
    corner = base[:1].copy()  # fixes the far end of the centroid box
    for f in ("p0", "p1", "p2"):
        corner[f] = np.float32(1.0) + corner[f] * np.float32(1e-3)
    parts.append(corner)
    return np.concatenate(parts)


def _levels(nodes):
    depth = np.zeros(len(nodes), np.int64)
    frontier, level = [0], 0
    while frontier:
        level += 1
        depth[frontier] = level
        ch = nodes["child"][frontier]
        used = ~np.isinf(nodes["lo_x"][frontier])
        frontier = ch[used & (ch >= 0)].tolist()
    assert (depth > 0).all()  # every node is reached, once per level list
    return level


@pytest.mark.parametrize("leaf,same", [(1, 40000), (4, 3000)])
def test_deep_trees(ctx, leaf, same):
    tris = _deep(leaf, same)
    scene = ctx.create_scene_gpu(tris, max_leaf_size=leaf)
    bvh = scene.download()  # validated: every record in one leaf, boxes, stack bounds
    levels = _levels(scene.read_bvh(LAYOUT_BVH4)[0])
    if leaf == 1:
        assert levels > WIDE_LEVELS
    rays = scenes.incoherent_rays(600, 7403, tmax=float(NO_HIT))
    rays["org"][::2] *= np.float32(0.05)
    expect, flags = pyoracle.trace_geometry(tris, rays)
    ok = (flags & pyoracle.EVENT_NAN_T) == 0
    got = scene.trace_geometry(rays)
    assert_hits_equal(got[ok], expect["prim"][ok], expect["t"][ok], expect["u"][ok], expect["v"][ok], f"leaf {leaf}",
                      rays=rays[ok], tris=tris)
    assert bvh.info["max_stack"] == scene.info["max_stack"]
