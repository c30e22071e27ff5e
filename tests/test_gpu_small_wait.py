"""A meeting of the small domain's step whose wait runs out (one CTA fewer is
launched than the meeting point counts): the kernel ends by itself, with status
bit 3, dt NaN and NaN in every depth that it was to write; the input stays; and
the next launch leaves at once instead of using the meeting point again."""
import math
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "swe-ppm_gb300", "csrc")
CELLS = 3 * 40


@pytest.fixture(scope="module")
def runs(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("wait") / "check")
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-fmad=false", "-std=c++17", "-I" + CSRC,
                    os.path.join(HERE, "gpu_small_wait_check.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    print(out)
    return {n: (int(status), float(dt), int(nans), int(left), int(changed), float(ms))
            for n, status, dt, nans, left, changed, ms in (line.split() for line in out.splitlines())}


def test_a_meeting_that_is_held(runs):
    status, dt, nans, left, changed, _ = runs["meets"]
    assert (status, nans, left, changed) == (0, 0, 0, 0) and 0 < dt < 1


def test_a_meeting_that_runs_out(runs):
    status, dt, nans, left, changed, _ = runs["runs_out"]
    assert status == 8 and math.isnan(dt)
    assert (nans, left, changed) == (CELLS, 0, 0)


def test_the_next_launch_leaves_at_once(runs):
    status, dt, nans, left, changed, ms = runs["again"]
    assert status == 8 and math.isnan(dt)
    assert (nans, left, changed) == (CELLS, 0, 0)
    assert ms < 0.1 * runs["runs_out"][5]
