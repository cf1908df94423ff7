"""Edge cases of the traversal on the kernels of large launches (one ray per lane).  Under the default launch
config launches of few rays run one warp per ray, so the other files' cases, small as they are, test that
kernel; here the same cases run again under a config that names the one-lane kernels: ties, equal t across
leaves, updates and refits, non-finite input, short rays, bounces, scenes, renders, host buffers, stack
overflow, the Lambertian schedule and its recovery from a deadline, and captured frames."""
import numpy as np
import pytest

import bvhtracer_gb300 as bt
from bvhtracer_gb300 import scenes
from test_gpu_adjoint import (test_forward_schedule_across_ray_counts_and_orders, test_lambert_forward_adjoint_against_fp64,  # noqa: F401
                              test_repeated_forward_passes_are_identical)
from test_gpu_deadline import (test_lambertian_forward_stops_and_its_schedule_recovers,  # noqa: F401
                               test_persistent_bounce_stops_at_the_deadline_and_recovers)
from test_gpu_frames import test_animated_frames_in_a_graph_match_the_oracle  # noqa: F401
from test_gpu_hidden import (test_bounce_kernels_with_hidden_trees, test_duplicate_triangles_in_different_hidden_leaves_tie_to_lowest_index,  # noqa: F401
                             test_equal_t_in_a_later_leaf_is_not_taken, test_flat_leaf_edges_vertices_and_random,
                             test_hidden_boxes_follow_vertex_updates_and_refit, test_instanced_scene_with_hidden_trees,
                             test_non_finite_vertices_and_odd_rays, test_reference_bvh_leaves_get_hidden_trees,
                             test_short_rays_stop_at_their_t)
from test_gpu_host_buffers import test_trace_bounce_with_every_kind_of_host_buffer  # noqa: F401
from test_gpu_in_place import case, test_host_buffers  # noqa: F401
from test_gpu_parity import (test_bounce_rays_and_hits, test_host_call_equals_device_launch, test_incoherent_rays_and_edge_cases,  # noqa: F401
                             test_near_tie_rays_counted_and_identical, test_render_shaders_match_oracle,
                             test_stack_overflow_is_reported_not_faulted, test_tlas_rebuild_and_scene_trace)
from test_gpu_render_scene import instanced, test_instanced_scene_render_matches_oracle  # noqa: F401

pytestmark = pytest.mark.gpu

KERNELS = (bt.K_TRACE_BLAS, bt.K_TRACE_SCENE, bt.K_PERSISTENT_BOUNCE, bt.K_SCENE_BOUNCE, bt.K_TRACE_BATCH)


class OneLane(bt.Context):
    def __init__(self, device=0):
        super().__init__(device)
        for k in KERNELS:
            self.tune_set(k, **dict(self.tune_get(k), big_leaf=17))


@pytest.fixture(scope="module", autouse=True)
def one_lane():
    with pytest.MonkeyPatch.context() as mp:
        mp.setattr(bt, "Context", OneLane)
        yield


@pytest.fixture(scope="module")
def ctx(one_lane):
    c = bt.Context(0)
    yield c
    c.close()


def test_the_config_is_not_the_default(ctx):
    assert type(ctx) is OneLane and all(ctx.tune_get(k)["big_leaf"] == 17 for k in KERNELS)


def test_lambertian_passes_of_both_kinds_alternate_on_one_mesh(ctx):
    """Warp-per-ray passes between scheduled ones: they neither read nor write the mesh's schedule."""
    verts, faces, vn, _, rays, light = scenes.lambert_scene(seed=6, level=7, width=200, height=200)
    n = len(rays)
    m = bt.DiffMesh(ctx, verts, faces, vn)
    d_rays, d_img, d_hits = ctx.to_device(rays), ctx.device_buffer(4 * n), ctx.device_buffer(bt.HIT.itemsize * n)
    d_back = ctx.to_device(np.ascontiguousarray(rays[::-1]))
    one = ctx.tune_get(bt.K_TRACE_BLAS)

    def forward(d, k):
        d_img.zero()
        d_hits.zero()
        m.forward_async(d, k, light, d_img, d_hits)
        ctx.sync()
        return d_img.download(np.zeros(n, np.float32)), d_hits.download(np.zeros(n, bt.HIT))

    try:
        img, hits = forward(d_rays, n)
        for i in range(8):
            ctx.tune_set(bt.K_TRACE_BLAS, **dict(one, big_leaf=16 if i % 3 == 1 else 17))  # 16: the default
            k = n if i % 4 else n // 2
            a, b = forward(d_back if i % 2 else d_rays, k)
            sel = slice(None, None, -1) if i % 2 else slice(None)
            assert a[:k].tobytes() == img[sel][:k].tobytes() and b[:k].tobytes() == hits[sel][:k].tobytes()
    finally:
        ctx.tune_set(bt.K_TRACE_BLAS, **one)
