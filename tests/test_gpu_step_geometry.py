"""The FP32 step kernel's dense staging geometry (three blocks on an SM) where
its tiles, runs and seams end: one tile in x, a short last run of planes, an odd
number of planes; against the oracle node by node, against z-slabs (whose ranges
of planes take the other geometry) bit for bit, and in the checked build.
test_step_plan.py pins that these boxes take it."""
from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from conftest import assert_state_close
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

KW = dict(rhoL=0.1, rhoH=1.0, tauRho=0.8, tauPhi=0.9, width=4.0, sigma=1e-3, Gamma=1.0)
BOXES = [(32, 96, 110), (96, 64, 95)]


def bubbles(shape):
    """One in the box, one through its x and z seams."""
    nx, ny, nz = shape
    return np.array([[0.5 * nx, 0.4 * ny, 0.4 * nz, 10.0], [1.3, 0.8 * ny, nz - 1.6, 7.0]], np.float32)


@pytest.mark.parametrize("shape", BOXES)
def test_dense_geometry_matches_the_oracle(lib, shape):
    from lbm_bench_gpu_gb300 import capi
    p = capi.make_params(*shape, **KW)
    o = Oracle.from_params(p)
    o.init_bubbles(bubbles(shape))
    with capi.Lattice.from_bubbles(p, bubbles(shape)) as lat:
        for n in (1, 1, 3):     # from the streamed state, odd, and further
            lat.step(n, -2e-5)
            o.step(n, -2e-5)
            assert_state_close(lat, o, what=f"dense {shape}")


@pytest.mark.parametrize("shape,depths", [((32, 96, 110), (53, 57)), ((96, 64, 95), (2, 78, 15))])
def test_dense_geometry_equals_slabs(lib, shape, depths):
    from lbm_bench_gpu_gb300 import capi
    p = capi.make_params(*shape, **KW)
    with capi.Lattice.from_bubbles(p, bubbles(shape)) as ref, capi.Lattice.from_bubbles(p, bubbles(shape)) as whole:
        with capi.Slabs(whole, depths) as slabs:
            slabs.step(7, -2e-5)
            slabs.merge_into(whole)
        ref.step(7, -2e-5)
        for a, b in zip(whole.dist(), ref.dist()):
            assert np.array_equal(a, b)
        fa, fb = whole.fields(), ref.fields()
        for k in fa:
            assert np.array_equal(fa[k], fb[k]), k


RUN = r"""
import sys
import numpy as np
from lbm_bench_gpu_gb300 import capi
sys.path.insert(0, sys.argv[1])
from test_gpu_step_geometry import BOXES, KW, bubbles
for shape in BOXES:
    p = capi.make_params(*shape, **KW)
    with capi.Lattice.from_bubbles(p, bubbles(shape)) as lat, capi.Slabs(lat, (shape[2] - 40, 40)) as slabs:
        slabs.step(5, -2e-5)
        slabs.stats()          # raises if the checked build flagged an index
        lat.step(5, -2e-5)
        lat.sync()
"""


def test_checked_build_flags_nothing(lib):
    from lbm_bench_gpu_gb300 import build
    env = dict(os.environ, LBM_GB300_LIB=str(build.build_checked()))
    r = subprocess.run([sys.executable, "-c", RUN, str(Path(__file__).parent)], cwd=Path(__file__).resolve().parents[1],
                       env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
