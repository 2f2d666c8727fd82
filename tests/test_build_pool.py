"""GPU-built scenes live in a memory pool of their context: scenes that come
and go on several streams and threads keep their own contents, and a scene
outlives its context."""
import math
import threading

import numpy as np
import pytest

import igx_raytracing_gb300 as igx
from igx_raytracing_gb300 import scenes

pytestmark = pytest.mark.gpu


def _tensor(a):
    import torch

    return torch.from_numpy(a.view(np.float32).reshape(len(a), -1).copy()).cuda()


def test_builds_on_streams_and_threads(ctx):
    import torch

    rays = scenes.incoherent_rays(3000, 7501)
    d_rays = _tensor(rays)
    sizes = [700, 40000, 5, 12000, 90000, 3]
    tris = [scenes.random_triangles(n, 7510 + n, mu=math.log(0.03)) for n in sizes]
    expect = []
    for t in tris:
        s = ctx.create_scene(t)
        expect.append(ctx.trace_closest(s, d_rays).cpu().numpy().view(np.uint32))
        s.close()
    d_tris = [_tensor(t) for t in tris]
    torch.cuda.synchronize()
    errors = []

    def work(k):
        try:
            stream = torch.cuda.Stream()
            live = []
            with torch.cuda.stream(stream):
                for i in range(12):
                    j = (k + i) % len(sizes)
                    s = ctx.create_scene_gpu(d_tris[j])
                    live.append((j, s, ctx.trace_closest(s, d_rays)))
                    if len(live) == 3:  # the oldest goes while two are alive
                        j, s, out = live.pop(0)
                        stream.synchronize()
                        if not np.array_equal(out.cpu().numpy().view(np.uint32), expect[j]):
                            errors.append((k, i, j))
                        s.close()
            stream.synchronize()
            for j, s, out in live:
                if not np.array_equal(out.cpu().numpy().view(np.uint32), expect[j]):
                    errors.append((k, j))
                s.close()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


def test_scene_outlives_its_context():
    rays = scenes.incoherent_rays(2000, 7502)
    tris = scenes.random_triangles(5000, 7503, mu=math.log(0.03))
    a, b = igx.Context(0), igx.Context(0)
    s = a.create_scene_gpu(tris)
    expect = s.trace_geometry(rays)
    a.close()
    got = b.trace_closest(s, _tensor(rays)).cpu().numpy().view(np.uint32).reshape(-1, 4)
    assert np.array_equal(got, expect.view(np.uint32).reshape(-1, 4))
    s.close()
    b.close()
