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
@pytest.mark.parametrize("n", [1, 2, 3, 64, 8192, 8193, 32768, 32769])
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
