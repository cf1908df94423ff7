"""The bottom-up refresh of the hidden trees at the edges of its shapes: smallest trees, blocks of 2 to 4
siblings, half-filled pairs, degenerate and non-finite triangles -- every record against the seal
restated over the node's own triangles (test_gpu_hidden.check_hidden_records), after the upload and after
updates, and again after an update that made everything finite."""
import numpy as np
import pytest

import bvhtracer_gb300 as bt
from bvhtracer_gb300 import scenes
from oracle import oracle as orc
from test_gpu_hidden import check_hidden_records, one_leaf_bvh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = bt.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n", [16, 17, 25, 33, 64, 129, 1000])
@pytest.mark.parametrize("kind", ["sphere", "soup"])
def test_records_after_upload_and_updates(ctx, n, kind):
    tris = (scenes.displaced_icosphere(4, 2).triangles() if kind == "sphere" else scenes.soup(2000, 4))[:n].copy()
    blas = ctx.upload_blas(one_leaf_bvh(tris), tris)
    check_hidden_records(blas, tris)
    for k in range(3):  # the arrival counters are back at zero after every refresh
        tris = (tris * np.float32(1.1) + np.float32(0.01 * k)).astype(np.float32)
        blas.update_vertices(tris)
        check_hidden_records(blas, tris)
    blas.free()


def test_degenerate_and_non_finite_triangles(ctx):
    good = scenes.displaced_icosphere(4, 2).triangles()[:200].copy()
    bad = good.copy()
    bad[3] = np.tile(bad[3, :3], 3)  # a point: no normal
    bad[50, 0] = np.nan
    bad[120, 5] = np.inf
    bad[180] = np.float32(1e20)
    blas = ctx.upload_blas(one_leaf_bvh(good), bad)
    with np.errstate(invalid="ignore"):
        check_hidden_records(blas, bad)
        blas.update_vertices(good)
        check_hidden_records(blas, good)
    blas.free()


def least_cosine(e1, e2, axis):
    """cone_terms (cull.cuh) restated in float32, operation by operation: the least lower bound of
    |N . A| / (|N| |A|) over the triangles."""
    f = np.float32
    u0 = f(2.0 ** -24)
    e1, e2 = e1.T, e2.T
    n, en = [], []
    for i, j in ((1, 2), (2, 0), (0, 1)):
        a, b = e1[i] * e2[j], e1[j] * e2[i]
        n.append(a - b)
        en.append(f(3) * u0 * (np.abs(a) + np.abs(b)))
    dot = err = nn = n_err = np.zeros(e1.shape[1], f)
    aa = f(0)
    for i in range(3):
        dot = dot + n[i] * axis[i]
        err = err + (en[i] + f(4) * u0 * np.abs(n[i])) * np.abs(axis[i])
        nn = nn + n[i] * n[i]
        n_err = n_err + en[i]
        aa = aa + axis[i] * axis[i]
    nlen, alen = np.sqrt(nn), np.sqrt(aa)
    one = f(1)
    num = np.abs(dot) - err
    den = (nlen * (one + f(8) * u0) + n_err) * alen * (one + f(8) * u0)
    n_lo = (nlen * (one - f(8) * u0) - n_err) * (one - f(4) * u0)
    return np.where((num > 0) & (den > 0) & (n_lo > 0), num / den * (one - f(8) * u0), f(-1)).min()


@pytest.mark.parametrize("n", [16, 17, 127, 129, 513, 5000, 20480])
@pytest.mark.parametrize("one", [True, False])
def test_root_cones_are_as_narrow_as_their_triangles(ctx, n, one):
    """In a large model a hidden root's cone is the one its triangles' normals span around its axis, bit for
    bit, after the upload and after updates: leaves of one root, of many, and warps that hold several."""
    tris = (scenes.displaced_icosphere(5, 2).triangles()[:n] * np.float32(100)).copy()
    bvh = one_leaf_bvh(tris) if one else bt.BvhBuilder().build_for(tris)
    blas = ctx.upload_blas(bvh, tris)
    leaves = [x for x in bvh.nodes[:bvh.nodes_used] if x["primitive_count"] >= 16]
    for k in range(3):
        if k:
            tris = (tris * np.float32([1.0, 1.0 + 0.2 * k, 1.0] * 3)).astype(np.float32)
            blas.update_vertices(tris)
        hd = blas.hidden_download()
        v = tris.reshape(-1, 3, 3)
        e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
        seen = 0
        for leaf in leaves:
            first, count = int(leaf["left_first"]), int(leaf["primitive_count"])
            cone = hd["cones"][int(hd["table"][first, 1]) & 0x0FFFFFFF]
            if cone[3] <= 0:
                assert not cone[:3].any()  # some normals lie square to the axis
                continue
            assert cone[3] == least_cosine(e1[first:first + count], e2[first:first + count], cone[:3])
            seen += 1
        assert seen >= (len(leaves) + 1) // 2 or (one and n > 100)
    blas.free()


@pytest.mark.parametrize("level,scale", [(3, 100.0), (5, 100.0), (5, 1.0)])
def test_mesh_update_measures_the_roots_in_its_refit(ctx, level, scale):
    """A mesh update refreshes, then measures a large model's root cones in the refit's pass over the
    triangles: the same cones as a vertex update of its own gives, and the oracle's refitted nodes, update after
    update and replayed from a graph; a small model's roots stay valid cones."""
    mesh = scenes.displaced_icosphere(level, 2)
    verts = (mesh.vertices * np.float32(scale)).astype(np.float32)
    m = bt.DiffMesh(ctx, verts, mesh.faces.astype(np.uint32), mesh.dirs.astype(np.float32))
    nodes0, used = m.bvh.nodes.copy(), m.bvh.nodes_used
    ctx.graph_begin()
    m.update_async()
    graph = ctx.graph_end()
    for k in range(4):
        verts = (verts * np.float32([1.0, 1.0 + 0.1 * k, 1.0])).astype(np.float32)
        m.set_vertices(verts)
        if k % 2:
            m.update_async()
        else:
            ctx.graph_launch(graph)
        ctx.sync()
        tris = np.ascontiguousarray(verts[m.faces].reshape(-1, 9), np.float32)
        check_hidden_records(m.blas, tris)
        ref = orc.bvh_refit(nodes0, used, tris)[:used]
        assert m.blas.download_nodes().tobytes() == ref.tobytes()
        fused = m.blas.hidden_download()["cones"]
        m.blas.update_vertices(tris)
        assert m.blas.hidden_download()["cones"].tobytes() == fused.tobytes()
        v = tris.reshape(-1, 3, 3)
        e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
        table = m.blas.hidden_download()["table"]
        leaves = [x for x in ref if x["primitive_count"] >= 16]
        assert leaves
        for leaf in leaves:
            first, count = int(leaf["left_first"]), int(leaf["primitive_count"])
            cone = fused[int(table[first, 1]) & 0x0FFFFFFF]
            if cone[3] > 0:
                least = least_cosine(e1[first:first + count], e2[first:first + count], cone[:3])
                assert cone[3] == least if scale > 1 else cone[3] <= least
    ctx.graph_free(graph)
    ctx.lib.bvhgpu_mesh_free(ctx.h, m.id)
    m.blas.free()
