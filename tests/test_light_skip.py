"""The specular powers that the point-light sum leaves out
(swegl_gb300/csrc/sgl_shade.cuh) change no sum: equal bits against the loop
that takes every power, with exponents over all that a material may hold and
bases around the threshold, on the host and (with the device's approximate
logarithm) on the GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    out = str(tmp_path_factory.mktemp("light_skip") / "light_skip")
    subprocess.run([nvcc, "-gencode=arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-fmad=false",
                    "-prec-div=true", "-prec-sqrt=true", "-ftz=false", "-Xcompiler", "-ffp-contract=off",
                    "-I", os.path.join(ROOT, "swegl_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "shade_math", "light_skip.cu"), "-o", out], check=True)
    return out


def check(exe, where, n):
    r = subprocess.run([exe, where, str(n)], capture_output=True, text=True, check=True)
    cases, diff, inside, beyond = map(int, r.stdout.split())
    assert cases == n
    assert inside > n // 10 and beyond > n // 20  # the threshold is reached on both sides of 1024
    assert diff == 0, f"{diff} of {cases} light sums differ from the loop that takes every power"


def test_skipped_powers_change_no_sum(exe):
    check(exe, "host", 2000000)


@pytest.mark.gpu
def test_skipped_powers_change_no_sum_on_the_device(exe):
    check(exe, "device", 1 << 28)
