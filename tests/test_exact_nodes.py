"""Scenes that stay on the exact nodes: which nodes launches trace, and the
kernels over the exact ones, which the default launches reach only where the
grid nodes (csrc/grid.cuh) cannot serve."""
import ctypes as C
import math

import numpy as np
import pytest

import igx_raytracing_gb300 as igx
from igx_raytracing_gb300 import scenes
from igx_raytracing_gb300._capi import HIT_DTYPE
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


def _far(tris):
    """One vertex far away: the grid's steps outgrow the other triangles."""
    out = tris.copy()
    out["p0"][7] += np.float32(3e6)
    return out


@pytest.mark.parametrize("starts_fit", [True, False])
def test_a_captured_batch_follows_its_scenes(ctx, starts_fit):
    """A batch's launch traces the grid nodes exactly while every scene's can
    serve, whichever way it was captured; an empty scene does not matter."""
    import torch

    a = scenes.random_triangles(3000, 8110, mu=math.log(0.03))
    b = scenes.random_triangles(500, 8111, mu=math.log(0.05))
    near, far = a, _far(a)
    scene, other, empty = ctx.create_scene(near if starts_fit else far), ctx.create_scene(b), ctx.create_scene(a[:0])
    rays = scenes.incoherent_rays(2000, 8112)
    d_rays = _device(rays)
    outs = [torch.empty(len(rays), 4, device="cuda") for _ in range(3)]
    batch = ctx.create_batch([(s, d_rays, None, o, 0) for s, o in zip((scene, other, empty), outs)])
    on_grid = lambda: bool(igx.lib().igxrt_internal_batch_uses_grid(batch._h))
    for step, t in enumerate([None, far, near, near, far, near]):
        if t is not None:
            scene.refit(_device(t))
        t = t if t is not None else (near if starts_fit else far)
        assert uses_grid(scene) == (t is near), step
        for o in outs:
            o.fill_(-1)
        batch.launch()
        assert on_grid() == (t is near), step
        torch.cuda.synchronize()
        for tri, o in zip((t, b, a[:0]), outs):
            got = o.cpu().numpy().view(HIT_DTYPE).reshape(-1)
            expect, flags = pyoracle.trace_geometry(tri, rays)
            for f in ("prim", "t", "u", "v"):
                assert np.array_equal(got[f][flags == 0].view(np.uint32), expect[f][flags == 0].view(np.uint32)), (step, f)
    batch.close()
    for s in (scene, other, empty):
        s.close()


def _overflowing(tris):
    """Two triangles whose distance along x is no float: the grid has no step
    there."""
    out = tris.copy()
    for k, x in ((3, -2.5e38), (4, 2.5e38)):
        out["p0"][k], out["p1"][k], out["p2"][k] = (x, 0, 0), (x, 1, 0), (x, 0, 1)
    return out


def test_a_captured_trace_over_a_range_that_overflows(ctx):
    """A trace captured over grid nodes keeps them: a refit whose range is no
    float takes that axis out of its box tests instead of losing hits."""
    import torch

    tris = scenes.random_triangles(500, 8115, mu=math.log(0.1))
    rays = scenes.incoherent_rays(2000, 8116)
    scene = ctx.create_scene(tris)
    d_rays, out = _device(rays), torch.empty(len(rays), 4, device="cuda")
    ctx.trace_closest(scene, d_rays, out=out)  # nothing is allocated in the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.trace_closest(scene, d_rays, out=out)
    for t, grid in ((tris, True), (_overflowing(tris), False), (tris, True)):
        scene.refit(_device(t))
        assert uses_grid(scene) == grid
        out.fill_(-1)
        graph.replay()
        torch.cuda.synchronize()
        got = out.cpu().numpy().view(HIT_DTYPE).reshape(-1)
        expect, flags = pyoracle.trace_geometry(t, rays)
        ok = flags == 0
        assert ok.mean() > 0.9 and (expect["prim"][ok] != 0xFFFFFFFF).mean() > 0.5
        for f in ("prim", "t", "u", "v"):
            assert np.array_equal(got[f][ok].view(np.uint32), expect[f][ok].view(np.uint32)), f
    scene.close()


@pytest.mark.parametrize("layout", [0, 1])
def test_a_batch_with_one_scene_off_the_grid(ctx, layout):
    """One launch traces one kind of nodes: a scene without usable grid nodes
    takes the batch to the exact ones, triangles and mixed, both query modes."""
    import torch

    sets = [scenes.random_triangles(n, 8120 + n, mu=math.log(0.04)) for n in (2000, 900, 3000)]
    sets[1] = _far(sets[1])
    live = [ctx.create_scene(t) for t in sets]
    assert [uses_grid(s) for s in live] == [True, False, True]
    rays = scenes.incoherent_rays(3000, 8121)
    d_rays = _device(rays)
    items, expect = [], []
    for s, t in zip(live, sets):
        for mode in (0, 1):
            out = (torch.full((len(rays),), 9, dtype=torch.int32, device="cuda") if mode
                   else torch.full((len(rays), 4), -1.0, device="cuda"))
            items.append((s, d_rays, None, out, mode))
            expect.append((pyoracle.trace_occlusion if mode else pyoracle.trace_geometry)(t, rays))
    batch = ctx.create_batch(items, params={"layout": layout})
    for launch in (batch.launch, lambda: ctx.trace_batch(items)):
        launch()
        torch.cuda.synchronize()
        for (_, _, _, out, mode), (want, flags) in zip(items, expect):
            ok = flags == 0
            if mode:
                assert np.array_equal(out.cpu().numpy().view(np.uint32)[ok], want[ok])
                out.fill_(9)
            else:
                got = out.cpu().numpy().view(HIT_DTYPE).reshape(-1)
                for f in ("prim", "t", "u", "v"):
                    assert np.array_equal(got[f][ok].view(np.uint32), want[f][ok].view(np.uint32)), f
                out.fill_(-1)
    assert not igx.lib().igxrt_internal_batch_uses_grid(batch._h)
    batch.close()
    for s in live:
        s.close()


def test_a_served_batch_with_one_scene_off_the_grid(ctx):
    """The server's table is rewritten for the exact nodes when a request over
    such a scene joins the batch, whatever was in it before."""
    sets = [scenes.random_triangles(n, 8130 + n, mu=math.log(0.04)) for n in (1500, 800)]
    sets[1] = _far(sets[1])
    live = [ctx.create_scene(t) for t in sets]
    assert [uses_grid(s) for s in live] == [True, False]
    srv = igx.Server(ctx, streams=1, slice_rays=700)
    ids = [srv.add_scene(s) for s in live]
    requests = []
    for k in range(24):  # fit ones first, so that a table is half filled
        which = 1 if k % 6 == 5 else 0
        rays = scenes.incoherent_rays(400 + 100 * k, 8140 + k)
        prev = np.where(np.arange(len(rays)) % 3 == 0, k, 0xFFFFFFFF).astype(np.uint32) if k % 2 else None
        requests.append((which, rays, prev, k % 3 == 2))
    tickets = [srv.submit(ids[w], r, p, int(m)) for w, r, p, m in requests]
    for t, (w, rays, prev, mode) in zip(tickets, requests):
        got = srv.wait(t)["out"]
        want, flags = (pyoracle.trace_occlusion if mode else pyoracle.trace_geometry)(sets[w], rays, prev)
        ok = flags == 0
        if mode:
            assert np.array_equal(got[ok], want[ok])
        else:
            for f in ("prim", "t", "u", "v"):
                assert np.array_equal(got[f][ok].view(np.uint32), want[f][ok].view(np.uint32)), f
    srv.close()
    for s in live:
        s.close()


@pytest.mark.parametrize("leaf", [1, 4, 16])
def test_ordinary_scenes_are_on_the_grid(ctx, leaf):
    for tris in (scenes.displaced_sphere(64, 32), scenes.random_triangles(4000, 8150), scenes.heightfield(40, 30, 8151)):
        scene = ctx.create_scene(tris, max_leaf_size=leaf)
        assert uses_grid(scene)
        scene.close()


def test_detail_below_the_grid_steps_stays_exact(ctx):
    from test_grid import _stadium

    scene = ctx.create_scene(_stadium(8160))
    assert not uses_grid(scene)
    scene.close()
