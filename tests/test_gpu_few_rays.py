"""Launches of few rays run one warp per ray (small leaves in order by the whole warp, large ones
through a warp-wide walk of their hidden tree): the hits equal the oracle's bit for bit at the edges
of that path -- ray counts around the warp, the block and both dispatch lines, leaf sizes around the
in-order limit, ties, a node list that overflows, odd rays and a deep tree."""
import numpy as np
import pytest

import bvhtracer_gb300 as bt
from bvhtracer_gb300 import scenes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = bt.Context(0)
    yield c
    c.close()


def one_leaf(tris):
    nodes = np.zeros(2, bt.NODE)
    v = tris.reshape(-1, 3)
    nodes[0]["bounds_min"], nodes[0]["bounds_max"] = v.min(0), v.max(0)
    nodes[0]["primitive_count"] = len(tris)
    return bt.Bvh(nodes, 2)


def check(ctx, bvh, tris, rays):
    blas = ctx.upload_blas(bvh, tris)
    got = blas.intersect(rays)
    ref = orc.bvh_intersect(bvh.nodes, bvh.nodes_used, tris, rays, threads=8)
    assert (got["prim"] == ref["prim"]).all() and got.tobytes() == ref.tobytes()
    blas.free()
    return ref


@pytest.mark.parametrize("mesh", ["soup", "sphere"])
@pytest.mark.parametrize("n", [1, 2, 3, 64, 8192, 8193, 32768, 32769])  # (lines of 1,000 and 5,120 triangles)
def test_ray_counts(ctx, mesh, n):
    tris = scenes.soup(1000, 3) if mesh == "soup" else scenes.displaced_icosphere(4, 3).triangles()
    bvh = bt.BvhBuilder().build_for(tris)
    rays = np.concatenate([scenes.sphere_rays((n + 1) // 2, 5, box=6.0),
                           scenes.look_at_rays(256, 256, (0, 0, -3.2), (0, 0, 0), 50.0)])[:n]
    check(ctx, bvh, tris, rays)


@pytest.mark.parametrize("count", [1, 15, 16, 63, 65, 511, 512, 513, 4097])
def test_leaf_sizes(ctx, count):
    tris = np.ascontiguousarray(scenes.displaced_icosphere(4, 9).triangles()[:count])
    ref = check(ctx, one_leaf(tris), tris, np.concatenate([
        scenes.sphere_rays(500, 6, box=3.0), scenes.look_at_rays(64, 64, (0, 3, -1), (0, 0, 0), 50.0)]))
    assert count < 511 or (ref["prim"] != bt.MISS).any()


def test_ties_short_rays_and_odd_directions(ctx):
    rng = np.random.default_rng(5)
    base = np.array([[-1, -1, 0, 1, -1, 0, 0, 1, 0]], np.float32)
    other = rng.uniform(-3, 3, (600, 9)).astype(np.float32)
    other[:, 2::3] += np.float32(4.0)
    tris = np.concatenate([other, np.repeat(base, 700, 0)])[rng.permutation(1300)]  # 700 exact copies
    tris = np.ascontiguousarray(tris)
    o = np.tile(np.array([0.05, -0.1, -5], np.float32), (40, 1))
    d = np.tile(np.array([0, 0, 1], np.float32), (40, 1))
    d[:20, :2] = rng.uniform(-0.05, 0.05, (20, 2))
    rays = orc.make_rays(o, d)
    rays["t"][30:] = np.float32(5.0)  # exactly the copies' distance: a hit needs t < 5
    odd = orc.make_rays([[0, 0, -10], [0, 0, -10], [0.1, 0.2, -10], [1e30, 0, 0], [0, 0, -5]],
                        [[1e-40, 0, 1], [-1e-30, 1e-38, 1], [0, 0, 0], [-1, 0, 0], [np.nan, 0, 1]])
    ref = check(ctx, one_leaf(tris), tris, np.concatenate([rays, odd]))
    copies = np.nonzero((tris == base[0]).all(1))[0]
    assert (ref["prim"][:20] == copies.min()).all()


def test_node_list_overflow_falls_back_to_the_ordered_test(ctx):
    """Thousands of coplanar slivers along one ray: more live hidden nodes than the warp's list holds."""
    k = 20000
    x = np.linspace(-1, 1, k, dtype=np.float32)
    tris = np.zeros((k, 3, 3), np.float32)
    tris[:, 0] = np.stack([x, np.full(k, -1, np.float32), np.zeros(k, np.float32)], 1)
    tris[:, 1] = tris[:, 0] + np.float32([0.2, 2, 0])
    tris[:, 2] = tris[:, 0] + np.float32([0, 2, 0.2])
    tris = np.ascontiguousarray(tris.reshape(k, 9))
    o = np.tile(np.float32([-5, 0, 0.05]), (16, 1))
    d = np.tile(np.float32([1, 0, 0]), (16, 1))
    d[:, 1] = np.linspace(-0.1, 0.1, 16)
    ref = check(ctx, one_leaf(tris), tris, orc.make_rays(o, d))
    assert (ref["prim"] != bt.MISS).any()


def around(limit):
    return [(1, 1), (7, 5), (limit // 128, 128), (limit // 128 + 1, 128)]


@pytest.mark.parametrize("level,limit", [(2, 16384), (4, 32768), (6, 65536)])
def test_bounce_render_and_lambert_lines(ctx, level, limit):
    """Both sides of the lines of the bounce, the renders and the Lambertian forward pass: the hits equal
    the oracle's, the images and intensities equal those of a set config (the one-thread kernels)."""
    mesh = scenes.displaced_icosphere(level, 5)
    big = scenes.Mesh(mesh.dirs, mesh.radius * 10.0, mesh.faces)
    for w, h in around(limit):
        rays = scenes.look_at_rays(w, h, (0, 1.0, -3.2), (0, 0, 0), 50.0)
        tris = mesh.triangles()
        bvh = bt.BvhBuilder().build_for(tris)
        blas = ctx.upload_blas(bvh, tris)
        ref0 = orc.bvh_intersect(bvh.nodes, bvh.nodes_used, tris, rays, threads=8)
        b, valid = orc.bounce_rays(rays, ref0, tris, 9)
        ref1 = np.zeros(len(rays), orc.HIT)
        ref1["t"], ref1["prim"], ref1["inst"] = np.finfo(np.float32).max, bt.MISS, bt.MISS
        if valid.any():
            ref1[valid] = orc.bvh_intersect(bvh.nodes, bvh.nodes_used, tris, b[valid], threads=8)
        h0, h1, n = blas.trace_bounce(rays, 9, bt.MODE_PERSISTENT)
        assert h0.tobytes() == ref0.tobytes() and h1.tobytes() == ref1.tobytes() and n == (ref0["prim"] != bt.MISS).sum()
        dm = bt.DiffMesh(ctx, big.vertices, big.faces.astype(np.uint32), big.dirs.astype(np.float32))
        far = scenes.look_at_rays(w, h, (0, 10.0, -32.0), (0, 0, 0), 50.0)
        d_rays, d_hits, d_img = ctx.to_device(far), ctx.device_buffer(20 * len(far)), ctx.device_buffer(4 * len(far))
        cam = bt.Camera.symmetric_fov(50.0, w / h, 0.1, 100.0, (0, 1.0, -3.2), (0, -0.298275, 0.954480), (-1, 0, 0),
                                      (0, 0.954480, 0.298275))
        saved = ctx.tune_get(bt.K_TRACE_BLAS)
        out = []
        try:
            for cfg in ({}, {"hidden": 500}):
                ctx.tune_set(bt.K_TRACE_BLAS, **cfg)
                dm.forward_async(d_rays, len(far), (20.0, 20.0, -30.0), d_img, d_hits)
                out.append(d_img.download(np.zeros(len(far), np.float32)).tobytes() +
                           d_hits.download(np.zeros(len(far), bt.HIT)).tobytes() +
                           blas.render(cam, w, h, bt.ACC_DEPTH, bt.SHADER_DEPTH, None, [1.0, 0.0])[0].tobytes())
        finally:
            ctx.tune_set(bt.K_TRACE_BLAS, **saved)
        assert out[0] == out[1]
        got = d_hits.download(np.zeros(len(far), bt.HIT))
        assert got.tobytes() == orc.bvh_intersect(dm.bvh.nodes, dm.bvh.nodes_used, dm.tris, far, threads=8).tobytes()
        blas.free()
        ctx.lib.bvhgpu_mesh_free(ctx.h, dm.id)
        dm.blas.free()


@pytest.mark.parametrize("n,level", [(1, 0), (3, 1), (40, 3), (300, 3)])
def test_scene_lines(ctx, n, level):
    """A scene's closest hits, bounces and image on both sides of its line against a set config, and the
    closest hits against the oracle."""
    tris = scenes.displaced_icosphere(level, 6).triangles().copy()
    bvh = bt.BvhBuilder().build_for(tris)
    blas = ctx.upload_blas(bvh, tris)
    blas.set_shading(normals=np.tile(np.float32([0, 0, 1]), (len(tris), 3)).reshape(len(tris), 9))
    rng = np.random.default_rng(n)
    xf = np.zeros((n, 16), np.float32)
    inv = np.zeros((n, 16), np.float32)
    for i in range(n):
        m = np.eye(4) * rng.uniform(0.5, 2.0)
        m[3, 3] = 1
        m[:3, 3] = rng.uniform(-6, 6, 3)
        xf[i] = m.T.reshape(16)
        inv[i] = np.linalg.inv(m).T.reshape(16)
    sc = ctx.scene([blas] * n, xf, inv)
    tl, used = sc.download_tlas()
    sa = orc.SceneArrays([(bvh.nodes[:bvh.nodes_used], bvh.nodes_used, tris)], np.zeros(n, np.int64), inv)
    total = n * len(tris)
    limit = 16384 if total < 4096 else 32768 if total < 65536 else 65536
    kernels = (bt.K_TRACE_SCENE, bt.K_SCENE_BOUNCE)
    saved = {k: ctx.tune_get(k) for k in kernels}
    for w, h in around(limit):
        rays = scenes.look_at_rays(w, h, (0, 1.0, -20.0), (0, 0, 0), 60.0)
        d_rays, d0, d1 = ctx.to_device(rays), ctx.device_buffer(20 * len(rays)), ctx.device_buffer(20 * len(rays))
        cam = bt.Camera((-0.6, 0.6, -0.4, 0.4, 1, 100), (0, 0, -20), (0, 0, 1), (1, 0, 0), (0, 1, 0))
        out = []
        try:
            for cfg in ({}, {"hidden": 500}):
                for k in kernels:
                    ctx.tune_set(k, **cfg)
                sc.trace_bounce_async(d_rays, len(rays), 5, d0, d1)
                hits = sc.intersect(rays)
                out.append(hits.tobytes() + d0.download(np.zeros(len(rays), bt.HIT)).tobytes() +
                           d1.download(np.zeros(len(rays), bt.HIT)).tobytes() +
                           sc.render(cam, w, h, bt.ACC_NORMAL, bt.SHADER_RADIANCE, lookup=bt.LOOKUP_HIT_OBJECT)[0].tobytes())
        finally:
            for k, v in saved.items():
                ctx.tune_set(k, **v)
        assert out[0] == out[1]
        assert hits.tobytes() == orc.scene_intersect(tl, used, sa, rays, threads=8).tobytes()
    sc.free()
    blas.free()


def test_default_and_set_configs_agree(ctx):
    tris = scenes.displaced_icosphere(5, 1).triangles()
    bvh = bt.BvhBuilder().build_for(tris)
    blas = ctx.upload_blas(bvh, tris)
    rays = scenes.sphere_rays(3000, 8, box=4.0)
    a = blas.intersect(rays)
    saved = ctx.tune_get(bt.K_TRACE_BLAS)
    try:
        ctx.tune_set(bt.K_TRACE_BLAS, hidden=500)  # a set config: the one-thread kernel
        assert blas.intersect(rays).tobytes() == a.tobytes()
    finally:
        ctx.tune_set(bt.K_TRACE_BLAS, **saved)


@pytest.mark.parametrize("n", [16384, 16385, 32768, 32769, 65536])
def test_scene_of_many_tiny_objects(ctx, n):
    """Many objects of 80 triangles: hits and bounces on both sides of their own lines, the closest hits
    against the oracle and the bounces against a set config."""
    tris = scenes.displaced_icosphere(1, 6).triangles().copy()
    bvh = bt.BvhBuilder().build_for(tris)
    blas = ctx.upload_blas(bvh, tris)
    k = 900
    rng = np.random.default_rng(k)
    xf = np.tile(np.eye(4, dtype=np.float32).reshape(1, 16), (k, 1))
    inv = xf.copy()
    xf[:, 12:15] = rng.uniform(-12, 12, (k, 3))
    inv[:, 12:15] = -xf[:, 12:15]
    sc = ctx.scene([blas] * k, xf, inv)
    tl, used = sc.download_tlas()
    sa = orc.SceneArrays([(bvh.nodes[:bvh.nodes_used], bvh.nodes_used, tris)], np.zeros(k, np.int64), inv)
    rays = np.concatenate([scenes.look_at_rays(128, 128, (0, 1.0, -40.0), (0, 0, 0), 45.0), scenes.sphere_rays(n, 3, box=14.0)])[:n]
    d_rays, d0, d1 = ctx.to_device(rays), ctx.device_buffer(20 * n), ctx.device_buffer(20 * n)
    saved = ctx.tune_get(bt.K_SCENE_BOUNCE)
    out = []
    try:
        for cfg in ({}, {"hidden": 500}):
            ctx.tune_set(bt.K_SCENE_BOUNCE, **cfg)
            sc.trace_bounce_async(d_rays, n, 5, d0, d1)
            out.append(d0.download(np.zeros(n, bt.HIT)).tobytes() + d1.download(np.zeros(n, bt.HIT)).tobytes())
    finally:
        ctx.tune_set(bt.K_SCENE_BOUNCE, **saved)
    assert out[0] == out[1]
    assert sc.intersect(rays).tobytes() == orc.scene_intersect(tl, used, sa, rays, threads=8).tobytes()
    sc.free()
    blas.free()
