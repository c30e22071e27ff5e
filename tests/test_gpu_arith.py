"""The edge arithmetic's operators for a known range (rcpRn, sqrtRn, divRn) and
the solvers' paths built on them against the general operators and paths, bit
for bit: every float of the unary operators' range, and hashed quotients and
edges.  The expected number of mismatches is 0; there is no tolerance."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "swe-ppm_gb300", "csrc")


@pytest.fixture(scope="module")
def counts(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("arith") / "check")
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-fmad=false", "-std=c++17", "-I" + CSRC,
                    os.path.join(HERE, "gpu_arith_check.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    return {n: (int(bad), int(of)) for n, bad, of in (line.split() for line in out.splitlines())}


@pytest.mark.parametrize("name", ["rcp", "sqrt", "div", "div_near", "fwave", "hlle", "augrie"])
def test_known_range_equals_general(counts, name):
    bad, of = counts[name]
    assert of > 0 and bad == 0, "%d of %d differ" % (bad, of)


def test_the_augmented_path_is_taken(counts):
    taken, of = counts["taken"]
    assert taken > of // 4  # (a check that never reaches the path would prove nothing)
