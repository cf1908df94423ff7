"""The TLAS rebuild's block variants (list in registers, 2 to 8 clusters a thread) against Tlas::rebuild
bit for bit, at the edges of every variant's range, with exact area ties, with empty boxes, and where the
reference would panic (no candidate below FLT_MAX)."""
import os
import subprocess
import sys

import numpy as np
import pytest

import bvhtracer_gb300 as bt
from bvhtracer_gb300 import scenes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def model():
    ctx = bt.Context(0)
    tris = scenes.displaced_icosphere(1, 5).triangles().copy()
    bvh = bt.BvhBuilder().build_for(tris)
    yield ctx, ctx.upload_blas(bvh, tris), bvh.nodes[0]
    ctx.close()


def placed(n, seed, grid):
    rng = np.random.default_rng(seed)
    xf = np.tile(np.eye(4, dtype=np.float32).reshape(16), (n, 1))
    inv = xf.copy()
    t = np.stack(np.unravel_index(rng.permutation(n), (17, 16, -(-n // 272))), 1) if grid else rng.uniform(-30, 30, (n, 3))
    xf[:, 12:15] = t
    inv[:, 12:15] = -xf[:, 12:15]
    return xf, inv


def check(model, xf, inv):
    ctx, blas, root = model
    n = len(xf)
    boxes = [orc.object_bounds(root["bounds_min"], root["bounds_max"], x) for x in xf]
    try:
        ref = orc.tlas_build(np.array([b[0] for b in boxes]), np.array([b[1] for b in boxes]))
    except RuntimeError:
        ref = None
    sc = ctx.scene([blas] * n)
    sc.set_transforms(xf, inv)
    if ref is None:
        with pytest.raises(bt.BvhGpuError):
            sc.rebuild()
    else:
        sc.rebuild()
        nodes, used = sc.download_tlas()
        assert used == ref[1] and nodes.tobytes() == ref[0].tobytes()
    sc.free()
    return ref


@pytest.mark.parametrize("grid", [False, True])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 127, 129, 256, 257, 512, 513, 1024, 1025, 2048, 2049, 4096])
def test_block_edges_and_ties(model, n, grid):
    assert check(model, *placed(n, n, grid)) is not None


@pytest.mark.parametrize("value", [np.nan, np.inf, 3e38, 1e19])
def test_boxes_without_a_finite_area(model, value):
    for n in (3, 300):
        xf, inv = placed(n, 7, False)
        xf[1, 12] = np.float32(value)
        check(model, xf, inv)


def test_nobody_left_to_merge_with(model):
    xf, inv = placed(5, 9, False)
    xf[:, 12] = np.array([-3e38, 3e38, -1e38, 2e38, 0], np.float32)
    assert check(model, xf, inv) is None


@pytest.mark.parametrize("n", [1532, 1533, 1536, 1537])
def test_sizes_at_the_default_shared_memory_limit(n):
    """1,533 objects fill 48 KB together with the block's own minima.  In a process of its own: a larger
    scene raises the kernel's limit for the rest of its process."""
    here = os.path.dirname(os.path.abspath(__file__))
    code = ("import bvhtracer_gb300 as bt\n"
            "from bvhtracer_gb300 import scenes\n"
            "from test_gpu_tlas_blocks import check, placed\n"
            "tris = scenes.displaced_icosphere(1, 5).triangles().copy()\n"
            "bvh = bt.BvhBuilder().build_for(tris)\n"
            "ctx = bt.Context(0)\n"
            f"assert check((ctx, ctx.upload_blas(bvh, tris), bvh.nodes[0]), *placed({n}, 3, False)) is not None\n")
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([os.path.dirname(here), here]))
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, env=env, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
