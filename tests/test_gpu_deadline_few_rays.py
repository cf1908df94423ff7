"""The launch deadline of launches that run one warp per ray: their warps start one after another, and the
budget counts from the launch's start, not from each warp's, so a launch longer than its budget stops even
where every single ray is far shorter -- also in a captured graph replayed under a deadline set later.
A launch without a deadline, or with a generous one, gives the same bytes as before."""
import time

import numpy as np
import pytest

import bvhtracer_gb300 as bt
from bvhtracer_gb300 import scenes

pytestmark = pytest.mark.gpu
N = 65536  # one warp per ray for models of this size, in several waves of warps
GENEROUS = 10 ** 10


@pytest.fixture(scope="module")
def ctx():
    c = bt.Context(0)
    yield c
    c.close()


def bounce(ctx):
    tris = scenes.displaced_icosphere(6, 3).triangles().copy()
    blas = ctx.upload_blas(bt.BvhBuilder().build_for(tris), tris)
    rays = scenes.look_at_rays(256, 256, (0, 0, -3.0), (0, 0, 0), 45.0)
    d, d0, d1 = ctx.to_device(rays), ctx.device_buffer(20 * N), ctx.device_buffer(20 * N)
    return lambda: blas.trace_bounce_async(d, N, 5, bt.MODE_PERSISTENT, d0, d1), (d0, d1), (blas, d)


def scene_bounce(ctx):
    tris = scenes.displaced_icosphere(3, 3).triangles().copy()
    blas = ctx.upload_blas(bt.BvhBuilder().build_for(tris), tris)
    xf = np.tile(np.eye(4, dtype=np.float32).reshape(1, 16), (500, 1))
    inv = xf.copy()
    xf[:, 12:15] = np.random.default_rng(1).uniform(-18, 18, (500, 3))
    inv[:, 12:15] = -xf[:, 12:15]
    sc = ctx.scene([blas] * 500, xf, inv)
    rays = scenes.look_at_rays(256, 256, (0, 0, -60.0), (0, 0, 0), 45.0)
    d, d0, d1 = ctx.to_device(rays), ctx.device_buffer(20 * N), ctx.device_buffer(20 * N)
    return lambda: sc.trace_bounce_async(d, N, 5, d0, d1), (d0, d1), (blas, sc, d)


def lambert(ctx):
    verts, faces, vn, _, rays, light = scenes.lambert_scene(seed=6, level=7, width=256, height=256)
    m = bt.DiffMesh(ctx, verts, faces, vn)
    d, img, hits = ctx.to_device(rays), ctx.device_buffer(4 * N), ctx.device_buffer(20 * N)
    return lambda: m.forward_async(d, N, light, img, hits), (img, hits), (m, d)


@pytest.mark.parametrize("make", [bounce, scene_bounce, lambert])
def test_budget_counts_from_the_launch(ctx, make):
    launch, outs, keep = make(ctx)

    def result():
        launch()
        ctx.sync()
        return [o.download(np.zeros(o.nbytes, np.uint8)).tobytes() for o in outs]

    ref = result()
    took = []
    for _ in range(5):
        t = time.perf_counter()
        for _ in range(20):
            launch()
        ctx.sync()
        took.append((time.perf_counter() - t) / 20)
    graph = None
    try:
        if make is bounce:
            ctx.graph_begin()
            launch()
            graph = ctx.graph_end()
        ctx.set_deadline(int(min(took) * 1e9 / 3))
        for _ in range(3):
            with pytest.raises(bt.BvhGpuError) as e:
                launch()
                ctx.sync()
            assert e.value.code == bt.ERR_DEADLINE
        if graph is not None:
            with pytest.raises(bt.BvhGpuError) as e:
                ctx.graph_launch(graph)
                ctx.sync()
            assert e.value.code == bt.ERR_DEADLINE
        ctx.set_deadline(GENEROUS)
        assert result() == ref
    finally:
        ctx.set_deadline(0)
    assert result() == ref
    if graph is not None:
        ctx.graph_launch(graph)
        ctx.sync()
        assert [o.download(np.zeros(o.nbytes, np.uint8)).tobytes() for o in outs] == ref
        ctx.graph_free(graph)
    del keep
