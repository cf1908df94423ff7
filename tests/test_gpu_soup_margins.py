"""Large leaves whose normals point everywhere (soups): rays whose margins are wide against the leaf test it
in order instead of walking its hidden tree, narrow ones walk it; hits are the oracle's bit for bit on both
sides of that rule and across it."""
import numpy as np
import pytest

import bvhtracer_gb300 as bt
from bvhtracer_gb300 import scenes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1000, 4096, 20000])
def test_wide_margins_test_a_soup_in_order(n):
    soup = scenes.soup(n, 3, scale=(n / 4096.0) ** (1 / 3))
    reach = 6.0 * (n / 4096.0) ** (1 / 3)
    entries = {}
    with bt.Context(0) as ctx:
        for k in (bt.K_TRACE_BLAS, bt.K_PERSISTENT_BOUNCE):  # any other config: one ray per lane at these counts
            ctx.tune_set(k, **dict(ctx.tune_get(k), big_leaf=17))
        for s in (0.5, 1.0, 1.4, 2.0, 3.0):
            tris = np.ascontiguousarray(soup * np.float32(s)).copy()
            bvh = bt.BvhBuilder().build_for(tris)
            rays = np.concatenate([scenes.look_at_rays(64, 64, (0, 0, -3 * s * reach), (0, 0, 0), 45.0),
                                   scenes.sphere_rays(4096, 7, box=2 * s * reach)])
            ref = orc.bvh_intersect(bvh.nodes, bvh.nodes_used, tris, rays, threads=8)
            blas = ctx.upload_blas(bvh, tris)
            assert blas.intersect(rays).tobytes() == ref.tobytes()
            h0, h1, _ = blas.trace_bounce(rays, 5, bt.MODE_PERSISTENT)
            second, valid = blas.bounce_rays(rays, 5)
            ref1 = orc.bvh_intersect(bvh.nodes, bvh.nodes_used, tris, second[valid], threads=8)
            assert h0.tobytes() == ref.tobytes() and h1[valid].tobytes() == ref1.tobytes()
            d_hits = ctx.device_buffer(bt.HIT.itemsize * len(rays))
            entries[s] = blas.trace_counts(ctx.to_device(rays), len(rays), d_hits)["hidden_entries"]
            blas.free()
    assert entries[0.5] > 100 and entries[3.0] < entries[0.5] / 10
