"""The boxes of posed primitives (swegl_gb300/csrc/sgl_cull.h, pose_box),
compiled for the host from the kernels' header: made from the boxes before the
transform, they hold every vertex as the pose pass transforms it (the whole-
primitive frustum test, which skips what cannot pass inside_camera_frustum,
src/render/renderer.cpp:58-70, relies on it), and boxes that are not finite
are marked.  Without the rounding margin the same vertices fall outside
thousands of times, so the inputs reach it."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("boxes", [200000])
def test_posed_boxes_hold_the_posed_vertices(tmp_path, boxes):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    out = str(tmp_path / "pose_box_host")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off",
                    "-I", os.path.join(ROOT, "swegl_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "shade_math", "pose_box_host.cu"), "-o", out], check=True)
    r = subprocess.run([out, str(boxes)], capture_output=True, text=True, check=True)
    n, vertices, outside, bare, unmarked = map(int, r.stdout.split())
    assert n == boxes and vertices > 10 * boxes
    assert outside == 0, f"{outside} of {vertices} vertices outside their posed box"
    assert unmarked == 0, f"{unmarked} boxes with an unbounded vertex are not marked"
    assert bare > 1000
