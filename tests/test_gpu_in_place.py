"""Closest hits from host arrays read and written in place: every kind of host buffer gives the oracle's
hits -- ordinary, page-locked, misaligned (staged), read-only rays, and a hit array that overlaps the
rays (staged) -- for one BLAS and for a scene, and an error leaves the context usable."""
import ctypes

import numpy as np
import pytest

import bvhtracer_gb300 as bt
from bvhtracer_gb300 import scenes
from bvhtracer_gb300._lib import ptr
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    ctx = bt.Context(0)
    tris = scenes.displaced_icosphere(4, 3).triangles().copy()
    bvh = bt.BvhBuilder().build_for(tris)
    blas = ctx.upload_blas(bvh, tris)
    eye = np.eye(4, dtype=np.float32).reshape(1, 16)
    yield ctx, blas, ctx.scene([blas], eye, eye), bvh, tris
    ctx.close()


@pytest.mark.parametrize("n", [1, 63, 5000, 40000])
@pytest.mark.parametrize("kind", ["ordinary", "pinned", "misaligned rays", "misaligned hits", "read-only", "overlap"])
def test_host_buffers(case, n, kind):
    ctx, blas, scene, bvh, tris = case
    rays = scenes.sphere_rays(n, n, box=2.0)
    ref = orc.bvh_intersect(bvh.nodes, bvh.nodes_used, tris, rays, threads=8)
    for call, handle in ((ctx.lib.bvhgpu_blas_intersect, blas.id), (ctx.lib.bvhgpu_scene_intersect, scene.id)):
        src, hits, keep = rays.copy(), np.zeros(n, bt.HIT), []
        p_rays, p_hits = ptr(src), ptr(hits)
        if kind == "pinned":
            a, b = ctx.pinned(n, bt.RAY), ctx.pinned(n, bt.HIT)
            a.array[:] = rays
            keep, hits = [a, b], b.array
            p_rays, p_hits = ptr(a.array), ptr(hits)
        elif kind == "misaligned rays":
            raw = np.zeros(32 * n + 64, np.uint8)
            off = (-raw.ctypes.data) % 16 + 4
            raw[off:off + 32 * n] = src.view(np.uint8)
            keep, p_rays = [raw], ctypes.c_void_p(raw.ctypes.data + off)
        elif kind == "misaligned hits":
            raw = np.zeros(20 * n + 64, np.uint8)
            off = (-raw.ctypes.data) % 4 + 1
            keep, p_hits = [raw], ctypes.c_void_p(raw.ctypes.data + off)
        elif kind == "read-only":
            src.flags.writeable = False
        elif kind == "overlap":
            p_hits = p_rays
        assert call(ctx.h, handle, p_rays, n, p_hits) == 0
        got = ctypes.string_at(p_hits, 20 * n)
        assert got == ref.tobytes()
        for x in keep:
            if isinstance(x, bt.PinnedArray):
                x.free()


def test_a_device_flag_is_reported_once(case):
    """The error flags travel with the call's last work: a failing call reports, the next one is clean."""
    ctx, _, _, _, _ = case
    n = 300
    nodes = np.zeros(2 + 2 * n, bt.NODE)  # a chain deeper than the largest traversal stack
    tris = np.tile(np.float32([-1, -1, 5, 1, -1, 5, 0, 1, 5]), (n + 1, 1))
    for i in range(n):
        k = 0 if i == 0 else 2 * i
        nodes[k]["bounds_min"], nodes[k]["bounds_max"], nodes[k]["left_first"] = -9, 9, 2 * i + 2
        for c in (2 * i + 2, 2 * i + 3):
            nodes[c]["bounds_min"], nodes[c]["bounds_max"] = -9, 9
        nodes[2 * i + 3]["primitive_count"], nodes[2 * i + 3]["left_first"] = 1, i
        nodes[2 * i + 3]["bounds_min"][2] = 4  # the leaf is the far child: it stays pending
    nodes[2 * n]["primitive_count"], nodes[2 * n]["left_first"] = 1, n
    blas = ctx.upload_blas(bt.Bvh(nodes, 2 * n + 2), tris)
    rays = orc.make_rays([[0, 0, -20]], [[0, 0, 1]])
    hits = np.zeros(1, bt.HIT)
    assert ctx.lib.bvhgpu_blas_intersect(ctx.h, blas.id, ptr(rays), 1, ptr(hits)) == 4
    ctx.sync()
    blas.free()
