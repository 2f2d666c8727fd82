"""The shadow pass's bookkeeping (csrc/shadow.cu: a group of 32 pairs keeps
its traced pairs and first slot, a warp packs four tile words): masks against
the oracle where the pairs or the words end inside a group, a block or a
warp's four words."""
import numpy as np
import pytest

from oracle import pyoracle
from test_shadow import shadow_setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(31, 1, 1), (32, 1, 1), (33, 1, 3), (17, 3, 1), (48, 2, 1), (80, 2, 1), (19, 27, 1),
                                  (61, 37, 2), (16, 34, 3)])
def test_masks(ctx, dims):
    w, h, s = dims
    tris, rays, obj = shadow_setup(w, h, s, seed=7900 + w + h)
    scene = ctx.create_scene(tris)
    for every in (1, 3):  # also with objects thinned out
        o = obj.copy()
        o[np.arange(len(o)) % every != 0] = 0xFFFFFFFF
        expect, flags = pyoracle.shadow_mask(tris, rays, o, w, h, s)
        assert not (flags & pyoracle.EVENT_NAN_T).any()
        assert np.array_equal(ctx.trace_shadow_mask(scene, rays, o, w, h, s), expect)
    scene.close()
