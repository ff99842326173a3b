"""The square root, reciprocal and quotient of the shader's normalisation on
the device: the root for every operand of its range, the quotients of every
significand of the length by 4,096 numerators, and by all of them for the
lengths whose reciprocal is a unit off (every pair: run the program with
8388608)."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_roots_reciprocals_and_quotients(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "normalize_roots_gpu")
    subprocess.run([nvcc, "-gencode=arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-fmad=false",
                    "-prec-div=true", "-prec-sqrt=true", "-ftz=false", "-I", os.path.join(ROOT, "swegl_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "shade_math", "normalize_roots_gpu.cu"), "-o", exe], check=True)
    r = subprocess.run([exe, "4096"], capture_output=True, text=True, check=True)
    roots, kept, kept_bad, pairs, bad = map(int, r.stdout.split())
    assert roots == 0 and kept_bad == 0 and bad == 0, r.stdout
    assert pairs == 1 << 35 and kept <= 4 * 200  # two significands of l, each from at most two s of an octave
