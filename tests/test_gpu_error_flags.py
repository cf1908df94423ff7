"""An error that a launch raises on the device is reported by that call alone: the next call succeeds with
the oracle's hits, also where the process has work queued on the default stream, and an error of its own is
not lost."""
import numpy as np
import pytest

import bvhtracer_gb300 as bt
from bvhtracer_gb300 import scenes
from bvhtracer_gb300._lib import ptr
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
STACK_DEPTH = 4  # BVHGPU_ERR_STACK_DEPTH


def too_deep(ctx, n=300):
    """A chain of nodes whose pending far children outgrow the largest traversal stack."""
    nodes = np.zeros(2 + 2 * n, bt.NODE)
    tris = np.tile(np.float32([-1, -1, 5, 1, -1, 5, 0, 1, 5]), (n + 1, 1))
    nodes["bounds_min"], nodes["bounds_max"] = -9, 9
    for i in range(n):
        nodes[0 if i == 0 else 2 * i]["left_first"] = 2 * i + 2
        nodes[2 * i + 3]["primitive_count"], nodes[2 * i + 3]["left_first"] = 1, i
        nodes[2 * i + 3]["bounds_min"][2] = 4  # the leaf is the far child: it stays pending
    nodes[2 * n]["primitive_count"], nodes[2 * n]["left_first"] = 1, n
    return ctx.upload_blas(bt.Bvh(nodes, 2 * n + 2), tris), orc.make_rays([[0, 0, -20]], [[0, 0, 1]])


@pytest.mark.parametrize("busy", [False, True])
def test_the_call_after_a_failed_one_is_clean(busy):
    torch = pytest.importorskip("torch")
    load = torch.zeros(1 << 28, device="cuda")
    tris = scenes.displaced_icosphere(4, 3).triangles().copy()
    bvh = bt.BvhBuilder().build_for(tris)
    rays = scenes.sphere_rays(100, 4, box=2.0)
    ref = orc.bvh_intersect(bvh.nodes, bvh.nodes_used, tris, rays)
    with bt.Context(0) as ctx:
        blas = ctx.upload_blas(bvh, tris)
        deep, down = too_deep(ctx)
        hit = np.zeros(1, bt.HIT)
        for _ in range(5):
            torch.cuda.synchronize()
            if busy:
                for _ in range(40):  # some milliseconds on the default stream
                    load.add_(1.0)
            for _ in range(2):  # twice: neither error is taken for the other's
                assert ctx.lib.bvhgpu_blas_intersect(ctx.h, deep.id, ptr(down), 1, ptr(hit)) == STACK_DEPTH
            assert blas.intersect(rays).tobytes() == ref.tobytes()
        torch.cuda.synchronize()
        ctx.sync()
