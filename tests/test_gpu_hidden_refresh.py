"""The bottom-up refresh of the hidden trees at the edges of its shapes: smallest trees, blocks of 2 to 4
siblings, half-filled pairs, degenerate and non-finite triangles -- every record against the seal
restated over the node's own triangles (test_gpu_hidden.check_hidden_records), after the upload and after
updates, and again after an update that made everything finite."""
import numpy as np
import pytest

import bvhtracer_gb300 as bt
from bvhtracer_gb300 import scenes
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
