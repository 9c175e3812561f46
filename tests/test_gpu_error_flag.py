"""A forward step whose bounded wait gave up sets the context's error flag and
leaves its tile unwritten: the calls that differentiate or sum over such states
report it.  The flag is set through the checked build's hook (a child process
loads that build), with no kernel that waits."""
from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

RUN = r"""
import ctypes as C, sys
import numpy as np
from lbm_bench_gpu_gb300 import capi
lib = capi.load()
lib.lbm_checked_raise_flag.argtypes = [C.c_void_p, C.c_int]
p = capi.make_params(32, 8, 8, rhoL=0.1, rhoH=1.0, tauRho=0.7, tauPhi=1.0, width=4.0, sigma=1e-3, Gamma=1.0)
calls = {"adjoint": lambda l: l.adjoint(3, -1e-5, "light_uz_mean", 2), "objective": lambda l: l.objective(3, -1e-5),
         "stats": lambda l: l.stats()}
for flag in (0, 1, 4):
    with capi.Lattice.from_bubbles(p, np.array([[15.0, 4.0, 4.0, 2.0]], np.float32)) as lat:
        assert lib.lbm_checked_raise_flag(lat._h, flag) == capi.LBM_OK
        try:
            calls[sys.argv[1]](lat)
            code = capi.LBM_OK
        except capi.LbmError as e:
            code = e.code
        print(flag, code, lat.steps)
"""


@pytest.mark.parametrize("call", ["adjoint", "objective", "stats"])
def test_calls_report_the_error_flag(lib, call):
    from lbm_bench_gpu_gb300 import build, capi
    env = dict(os.environ, LBM_GB300_LIB=str(build.build_checked()))
    r = subprocess.run([sys.executable, "-c", RUN, call], cwd=Path(__file__).resolve().parents[1], env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    want = {0: capi.LBM_OK, 1: capi.LBM_ETIMEOUT, 4: capi.LBM_ECUDA}
    assert [tuple(map(int, line.split())) for line in r.stdout.split("\n") if line] == [(f, c, 0) for f, c in want.items()]
