"""The library's host sources on a stand-in for the CUDA runtime
(tests/host_runtime): streams that execute nothing until something waits for
them, so that a missing wait shows without a GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "swegl_gb300", "csrc")
HERE = os.path.join(ROOT, "tests", "host_runtime")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("CUDA headers not available")
    out = str(tmp_path_factory.mktemp("host_runtime") / "host_runtime")
    src = [os.path.join(HERE, f) for f in ("host_runtime.cpp", "fake_cuda.cpp")]
    src += [os.path.join(CSRC, f) for f in ("sgl_api.cpp", "sgl_lane.cpp", "sgl_scene.cpp", "sgl_serve.cpp")]
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-I", HERE,
                    "-I", cuda, *src, "-lpthread", "-o", out], check=True)
    return out


def run(exe, scenario):
    r = subprocess.run([exe, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    return [int(x) for x in r.stdout.split()]


def test_calls_on_alternating_streams_are_ordered(exe):
    """A context's device calls share their scratch, so a call on another
    stream starts after the one before."""
    (unordered,) = run(exe, "streams")
    assert unordered == 0


def test_only_own_streams_are_destroyed(exe):
    foreign, twice = run(exe, "ownership")
    assert foreign == 0 and twice == 0


def test_staging_is_not_reused_before_its_copy_after_a_failed_call(exe):
    dof, batches, posed = run(exe, "failures")
    assert (dof, batches, posed) == (0, 0, 0)


def test_a_request_stays_within_the_budget_that_admits_it(exe):
    over = run(exe, "budget")
    assert len(over) == 4 and max(over) <= 0


def test_upload_allocates_and_launches_no_more_than_it_needs(exe):
    """15 arrays, 12 copies, one launch sequence."""
    (calls,) = run(exe, "uploads")
    assert calls <= 28
