"""The margins of the in-leaf cull (csrc/cull.cuh) against the float test's true errors.

tests/cull_margins.cpp is compiled with the library's own header (no fused multiply-add) and measures,
for triangles the float test accepts, how far the exact intersection lies from the computed one: it
must lie within the margins that leaf_cull grows the boxes by.  Margins shrunk 20 times must be
caught, which shows that the inputs reach errors of the margins' own order."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def margins(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("cull") / "cull_margins")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "bvhtracer_gb300", "csrc"), os.path.join(ROOT, "tests", "cull_margins.cpp"),
                    "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("scale", [1.0, 0.05])
def test_exact_intersection_lies_within_the_margins(margins, scale):
    out = subprocess.run([margins, "3000000", str(scale)], capture_output=True, text=True).stdout
    m = re.search(r"accepted (\d+) low-det (\d+) coned (\d+) violations (\d+)", out)
    assert m, out
    accepted, low_det, coned, violations = (int(x) for x in m.groups())
    assert accepted > 1_000_000 and low_det > 10_000 and coned > 300_000
    assert violations == 0 if scale == 1.0 else violations > 0, out
