"""Scenes that stay on the exact nodes: which nodes launches trace, and the
kernels over the exact ones, which the default launches reach only where the
grid nodes (csrc/grid.cuh) cannot serve."""
import ctypes as C
import math

import numpy as np
import pytest

import igx_raytracing_gb300 as igx
from igx_raytracing_gb300 import scenes
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def uses_grid(scene) -> bool:
    return bool(igx.lib().igxrt_internal_uses_grid(scene.handle))


def limited(records: int):
    """A context whose scenes of more records stay on the exact nodes."""
    c = igx.Context(0)
    igx.lib().igxrt_internal_set_grid_records(c.handle, C.c_uint64(records))
    return c


def _device(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a).view(np.float32).reshape(len(a), -1).copy()).cuda()


def _check(scene, tris, rays, what):
    hits = scene.trace_geometry(rays)
    expect, flags = pyoracle.trace_geometry(tris, rays)
    ok = flags == 0
    assert ok.mean() > 0.5
    for f in ("prim", "t", "u", "v"):
        a, b = hits[f][ok].view(np.uint32), expect[f][ok].view(np.uint32)
        assert np.array_equal(a, b), f"{what}: {f} differs on {(a != b).sum()} of {ok.sum()} rays"


@pytest.mark.parametrize("gpu_build", [False, True])
def test_a_refit_keeps_a_scene_too_large_for_the_references(gpu_build):
    """A grid leaf names its first record in 27 bits: a scene with more records
    has no grid nodes, before and after its refits."""
    ctx = limited(1000)
    for n, grid in ((1000, True), (1001, False)):
        tris = scenes.random_triangles(n, 8100 + n, mu=math.log(0.05))
        scene = ctx.create_scene_gpu(_device(tris)) if gpu_build else ctx.create_scene(tris)
        rays = scenes.incoherent_rays(1500, 8103)
        assert uses_grid(scene) == grid
        moved = tris.copy()
        for f in ("p0", "p1", "p2"):
            moved[f] = tris[f] * np.float32(0.9)
        for t in (moved, tris):
            scene.refit(_device(t))
            assert uses_grid(scene) == grid, f"{n} records after a refit"
            _check(scene, t, rays, f"{n} records")
        scene.close()
    ctx.close()
