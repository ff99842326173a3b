"""The shader's normalisation with one reciprocal square root, on the device,
against square root and divisions: equal bits on 2^30 seeded vectors (ordinary
ones, exponents across both ends of its range, zeros, subnormals, infinities
and NaNs)."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_normalize_fast_equals_square_root_and_divisions(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "normalize_gpu")
    subprocess.run([nvcc, "-gencode=arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-fmad=false",
                    "-prec-div=true", "-prec-sqrt=true", "-ftz=false", "-I", os.path.join(ROOT, "swegl_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "shade_math", "normalize_gpu.cu"),
                    "-o", exe], check=True)
    r = subprocess.run([exe, str(1 << 30)], capture_output=True, text=True, check=True)
    vectors, bad = map(int, r.stdout.split())
    assert vectors == 1 << 30 and bad == 0, f"{bad} of {vectors} vectors differ"
