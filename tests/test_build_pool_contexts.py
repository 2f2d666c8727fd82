"""Pools of several contexts at once: a context belongs to one host thread at a
time, so each thread builds, traces and destroys scenes in its own, on a stream
of its own."""
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


def test_builds_in_a_context_per_thread(ctx):
    import torch

    d_rays = _tensor(scenes.incoherent_rays(3000, 8501))
    sizes = [700, 40000, 5, 12000, 90000, 3]
    tris = [scenes.random_triangles(n, 8510 + n, mu=math.log(0.03)) for n in sizes]
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
            own = igx.Context(0)
            stream = torch.cuda.Stream()
            live = []

            def retire():
                j, s, out = live.pop(0)
                stream.synchronize()
                if not np.array_equal(out.cpu().numpy().view(np.uint32), expect[j]):
                    errors.append((k, j))
                s.close()

            with torch.cuda.stream(stream):
                for i in range(12):
                    j = (k + i) % len(sizes)
                    s = own.create_scene_gpu(d_tris[j])
                    live.append((j, s, own.trace_closest(s, d_rays)))
                    if len(live) == 3:  # the oldest goes while two are alive
                        retire()
                while live:
                    retire()
            own.close()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
