"""The device planning of the hidden trees: every triangle of a large leaf in exactly one pair slot, leaves
of 1 to 8 triangles, nodes of 2 to 4 children each reached once, the same plan for the same triangles, and
hits equal to the oracle's -- at the sizes where the block's passes and the level loop change, for
coinciding centroids (halves by order), coordinates over many orders of magnitude (uneven splits,
deep trees) and several leaves of which some are too small."""
import numpy as np
import pytest

import bvhtracer_gb300 as bt
from bvhtracer_gb300 import scenes
from oracle import oracle as orc
from test_gpu_hidden import one_leaf_bvh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = bt.Context(0)
    yield c
    c.close()


def check_plan(blas, big):
    """`big`: the triangle indices of the large leaves, one array per leaf."""
    hd, h = blas.hidden_download(), blas.hidden()
    ui, base, p0 = hd["nodes"].view(np.uint32), blas.nodes_used, (blas.ntris + 1) // 2
    roots = np.nonzero(hd["table"][:, 1])[0]
    assert sorted(roots) == sorted(b[0] for b in big)
    seen_nodes, seen_pairs, deepest = set(), set(), 0
    for leaf in big:
        got = []
        todo = [(int(hd["table"][leaf[0], 0]), int(hd["table"][leaf[0], 1]), 0)]
        while todo:
            first, count, depth = todo.pop()
            deepest = max(deepest, depth)
            if count & 0x80000000:
                n = count & 0x7FFFFFFF
                assert 1 <= n <= 4
                for p in range(first - p0, first - p0 + n):
                    assert p not in seen_pairs
                    seen_pairs.add(p)
                    got += [int(t) for t in hd["slots"][p] if t != 0xFFFFFFFF]
                continue
            assert count & 0x40000000
            for c in range(first - base, first - base + ((count >> 28) & 3) + 1):
                assert c not in seen_nodes
                seen_nodes.add(c)
                todo.append((int(ui[c, 3]), int(ui[c, 7]), depth + 1))
        assert sorted(got) == sorted(leaf)
    assert len(seen_nodes) == h["nodes"] and len(seen_pairs) == h["pairs"] and deepest == h["depth"]


def trace(blas, bvh, tris, seed, box):
    rays = scenes.sphere_rays(3000, seed, box=box)
    ref = orc.bvh_intersect(bvh.nodes, bvh.nodes_used, tris, rays, threads=8)
    assert blas.intersect(rays).tobytes() == ref.tobytes()


def shapes(kind, n):
    if kind == "sphere":
        return scenes.displaced_icosphere(5, 6).triangles()[:n].copy()
    if kind == "same":  # every centroid the same: no split plane
        return np.tile(scenes.soup(1, 3), (n, 1))
    rng = np.random.default_rng(n)  # centroids from 1e-3 to 1e6 along x
    t = rng.uniform(-1, 1, (n, 3, 3))
    t[:, :, 0] += (10.0 ** rng.uniform(-3, 6, n))[:, None]
    return np.ascontiguousarray(t.reshape(n, 9).astype(np.float32))


@pytest.mark.parametrize("kind", ["sphere", "same", "spread"])
@pytest.mark.parametrize("n", [15, 16, 17, 64, 65, 511, 513, 1025, 5000])
def test_one_leaf(ctx, kind, n):
    tris = shapes(kind, n)
    bvh = one_leaf_bvh(tris)
    blas = ctx.upload_blas(bvh, tris)
    check_plan(blas, [np.arange(n)] if n >= 16 else [])
    trace(blas, bvh, tris, n, 4.0)
    again = ctx.upload_blas(bvh, tris)
    a, b = blas.hidden_download(), again.hidden_download()
    assert all(a[k].tobytes() == b[k].tobytes() for k in a)
    blas.free()
    again.free()


@pytest.mark.parametrize("n", [300, 4096, 30000])
def test_leaves_of_a_built_bvh(ctx, n):
    tris = scenes.soup(n, 8, scale=(n / 4096.0) ** (1 / 3))
    bvh = bt.BvhBuilder().build_for(tris)
    blas = ctx.upload_blas(bvh, tris)
    nodes = bvh.nodes[:bvh.nodes_used]
    leaves = nodes[(nodes["primitive_count"] >= 16)]
    check_plan(blas, [np.arange(l["left_first"], l["left_first"] + l["primitive_count"]) for l in leaves])
    trace(blas, bvh, tris, n, 12.0)
    blas.free()


@pytest.mark.parametrize("kind", ["sphere", "spread"])
def test_queued_levels_and_staging_memory(kind):
    """Around the sizes up to which the levels are queued ahead and the work area is the context's staging
    memory, in one fresh context and mixed with host traces that use and grow that memory; the models
    uploaded first keep their hits."""
    kept = []
    with bt.Context(0) as ctx:
        for n in (2048, 40, 2049, 4096, 16, 4097, 2047, 4095):
            tris = shapes(kind, n)
            bvh = one_leaf_bvh(tris)
            blas = ctx.upload_blas(bvh, tris)
            check_plan(blas, [np.arange(n)])
            kept.append((blas, bvh, tris))
            ctx.trace_batch(np.array([(blas.id, 0, 60000, 0)], bt.BATCH_ITEM), scenes.sphere_rays(60000, n, box=4.0), bt.MODE_PLAIN)
        for blas, bvh, tris in kept:
            trace(blas, bvh, tris, 5, 4.0)
