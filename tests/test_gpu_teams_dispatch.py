"""The update pass in CTAs of four teams against the pass in CTAs of one, bit for
bit, with the launches counted: a partition into exactly four runs per SM (the
default one of these domains) takes the first, shorter segments, and so more
runs, the second.  In a process with a library in front of the CUDA runtime's
launch call."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
PRODUCT = os.path.join(os.path.dirname(HERE), "swe-ppm_gb300")

DRIVE = """
import ctypes, sys
sys.path[:0] = [%r, %r]
import numpy as np
import swe_gb300 as swe
from helpers import assert_bitwise
from test_gpu_teams import waves
log = ctypes.CDLL(None)

def run(make, st, drive):
    D = make()
    D.upload(*st)
    D.exchange_bathymetry()
    c = (ctypes.c_int * 2)()
    log.launchCounts(c)
    drive(D)
    log.launchCounts(c)
    assert D.status() == 0
    out = D.download() + ((D.lts_state()[3],) if drive is interval else D.group_state())
    D.close()
    return out, c[0], c[1]

def interval(D):
    D.lts_advance(1.5)

def both(name, columns, make, st, drive):
    short = max(1, columns // 1000)  # segments that need more than four runs per SM
    a, four, _ = run(lambda: make(0), st, drive)
    r, none, one = run(lambda: make(short), st, drive)
    for i, (x, y) in enumerate(zip(a, r)):
        assert_bitwise(np.asarray(x), np.asarray(y), "%%s: output %%d" %% (name, i))
    print(name, four, none, one, flush=True)

for nx, ny, nb in ((2500, 256, 1), (1100, 769, 1), (1300, 1280, 4), (2048, 2048, 16), (9000, 1024, 1)):
    geo, st = waves(swe, nx, ny, nb, nx)
    cols, rows = geo["nx_cols"], geo["ny_rows"]
    columns = sum(-(-r // 256) for r in rows) * sum(cols)
    for solver in (1, 4):
        both("%%dx%%d/%%d" %% (nx, ny, nb), columns,
             lambda c: swe.Domain(cols, rows, geo["dx"], geo["dy"], boundary=[0, 1, 1, 0], solver=solver, tile_cols=c,
                                  tile_rows=256), st, lambda D: D.step(4))

inst, st = [], [[], [], [], []]
for i, (nx, ny) in enumerate([(700, 256), (900, 512), (650, 256), (800, 1024)]):
    geo, f = waves(swe, nx, ny, 1, i)
    inst.append((nx, ny, 2.0 + 3.0 * i, 5.0, [1, 0, 0, 1]))
    for a, v in zip(st, f):
        a.append(v)
both("stopped_groups", 700 + 1800 + 650 + 3200, lambda c: swe.Ensemble(inst, solver=4, tile_cols=c, tile_rows=256),
     [np.concatenate(a) for a in st], lambda D: D.advance(0.6))

geo, st = waves(swe, 2048, 1024, 8, 2)
both("lts", 4 * 2048, lambda c: swe.Domain(geo["nx_cols"], geo["ny_rows"], geo["dx"] * 20, geo["dx"] * 20, boundary=[1] * 4,
                                           solver=4, tile_cols=c, tile_rows=256, lts_max_timestep=1.0, duration=100.0),
     st, interval)
"""


def test_four_teams_equal_one_and_are_taken(swe, tmp_path):
    so = str(tmp_path / "liblaunchlog.so")
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-I/usr/local/cuda/include", os.path.join(HERE, "launch_log.cpp"),
                    "-o", so, "-ldl"], check=True)
    out = subprocess.run([sys.executable, "-c", DRIVE % (PRODUCT, HERE)], check=True, stdout=subprocess.PIPE, text=True,
                         timeout=300, env=dict(os.environ, LD_PRELOAD=so)).stdout
    runs = [line.split() for line in out.splitlines()]
    assert len(runs) == 12
    for name, four, none, one in runs:
        others = 0 if name != "lts" else int(none)  # (the check of local time stepping has CTAs of 1024 threads too)
        assert int(none) == others and int(four) - others >= 4 and int(one) >= 4, (name, four, none, one)
