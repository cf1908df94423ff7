"""The autotuner and a margin limit above its candidates: kept where it is clearly the fastest, as for a model in
large units, whose rays walk its hidden trees under margins of more than one triangle."""
import numpy as np
import pytest

import bvhtracer_gb300 as bt
from bvhtracer_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_a_wide_limit_survives_where_it_pays():
    tris = np.ascontiguousarray(scenes.displaced_icosphere(5, 3).triangles() * np.float32(30)).copy()
    rays = scenes.look_at_rays(400, 400, (0, 0, -90.0), (0, 0, 0), 45.0)
    with bt.Context(0) as ctx:
        blas = ctx.upload_blas(bt.BvhBuilder().build_for(tris), tris)
        d_rays, d0, d1 = ctx.to_device(rays), ctx.device_buffer(20 * len(rays)), ctx.device_buffer(20 * len(rays))
        assert ctx.tune_get(bt.K_PERSISTENT_BOUNCE)["hidden"] == 2000
        blas.trace_bounce_async(d_rays, len(rays), 5, bt.MODE_PERSISTENT, d0, d1)
        ref = d0.download(np.zeros(len(rays), bt.HIT)).tobytes()
        cfg, ms = ctx.autotune(bt.K_PERSISTENT_BOUNCE, d_rays, len(rays), d0, d1, target=blas.id, seed=5, reps=3)
        assert cfg["hidden"] == 2000 and cfg == ctx.tune_get(bt.K_PERSISTENT_BOUNCE) and ms > 0
        blas.trace_bounce_async(d_rays, len(rays), 5, bt.MODE_PERSISTENT, d0, d1)
        assert d0.download(np.zeros(len(rays), bt.HIT)).tobytes() == ref
