"""Steps that would go out as one cooperative launch where that launch cannot
run: on a stream of a green context (a part of the device's SMs, on which an
oversized cooperative launch never starts) none is tried, and where one is
refused the passes take its place.  On the CPU, against a stand-in for the CUDA
runtime that records the launches."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PRODUCT = os.path.join(os.path.dirname(HERE), "swe-ppm_gb300")

DRIVE = """
import ctypes, sys
sys.path.insert(0, %r)
import swe_gb300 as swe
fake = ctypes.CDLL(None)
fake.fakeLaunches.restype = ctypes.c_char_p

def launched(refuse, green, call):
    fake.fakeSet(refuse, green)
    call()
    return fake.fakeLaunches().decode()

def block():
    swe.step_block_noalloc(swe.HLLE, swe.UNSPLIT, 64, 64, 1.0, 1.0, [1] * 4, 66, [16] * 4, [16] * 3, want_dt=False)

D = swe.Domain([64], [64], 1.0, 1.0, solver=swe.HLLE)
D.step(1)  # (sets the ghost ring)
for refuse, green in ((0, 0), (1, 0), (0, 1)):
    fake.fakeSet(refuse, green)
    D.set_stream(0x400)
    print(launched(refuse, green, block), launched(refuse, green, lambda: D.step(3)),
          launched(refuse, green, lambda: D.advance(1e30, max_steps=17)))
"""


@pytest.fixture(scope="module")
def lines(swe, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-I/usr/local/cuda/include", os.path.join(HERE, "fake_cudart.cpp"), "-o", so],
                   check=True)
    out = subprocess.run([sys.executable, "-c", DRIVE % PRODUCT], check=True, capture_output=True, text=True, timeout=120,
                         env=dict(os.environ, LD_PRELOAD=so)).stdout
    return [line.split() for line in out.splitlines()]


def test_one_cooperative_launch_where_it_can_run(lines):
    block, step, advance = lines[0]
    assert block == "kc"            # set-up, the step
    assert step == "c"              # three steps
    assert advance == "kck"         # target, seventeen steps, target


def test_a_refused_launch_is_replaced_by_the_passes(lines):
    block, step, advance = lines[1]
    assert block == "krkk"          # speed and update pass in the step's place
    assert step == "r" + "kk" * 3
    assert advance == "kr" + "kk" * 17 + "k"


def test_no_cooperative_launch_on_a_part_of_the_device(lines):
    block, step, advance = lines[2]
    assert block == "kkk"
    assert step == "kk" * 3
    assert advance == "[" + "kk" * 16 + "]kg" + "kk" + "k"
