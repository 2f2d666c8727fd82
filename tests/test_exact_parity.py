"""The parity tests of the queries and passes once more, over scenes that stay
on the exact nodes: every other launch that names BVH2 or BVH4 traces the grid
nodes, so the kernels over the exact layouts run only where those cannot
serve.  The same tests, with a context whose scenes get no grid nodes."""
import pytest

from test_batch_gpu import test_graph_batch_replays_identically, test_trace_batch_matches_plain  # noqa: F401
from test_exact_nodes import limited, uses_grid
from test_gbuffer import test_gbuffer_device_memory, test_gbuffer_matches_oracle  # noqa: F401
from test_mixed import test_gpu_mixed_golden, test_gpu_mixed_matches_oracle  # noqa: F401
from test_mixed_passes import (test_batch_with_mixed_scenes_matches_oracle,  # noqa: F401
                               test_gbuffer_mixed_matches_oracle, test_plain_queries_on_mixed_scenes_many_seeds,
                               test_server_serves_mixed_scenes_like_the_oracle,
                               test_shadow_mask_mixed_matches_oracle)
from test_refit import test_gpu_refit_mixed, test_gpu_refit_traces_match_oracle  # noqa: F401
from test_shadow import test_shadow_mask_device_memory, test_shadow_mask_matches_oracle  # noqa: F401
from test_trace_gpu import (params, test_golden_closest_host_memory, test_golden_device_memory,  # noqa: F401
                            test_interval_semantics, test_launch_shapes_agree, test_single_triangle_scene,
                            test_small_workload_all_rays_vs_brute_force)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = limited(0)
    yield c
    c.close()


def test_no_scene_of_the_context_is_on_the_grid(ctx):
    from igx_raytracing_gb300 import scenes

    for scene in (ctx.create_scene(scenes.random_triangles(500, 1)),
                  ctx.create_scene_gpu(scenes.random_triangles(500, 1))):
        assert not uses_grid(scene)
        scene.close()
