"""dJ/dphi0 of the u_z objective with a BF16 state against the oracle's FP64
adjoint, over an averaging window.  The nodes that may stand on the other side
of H(phi > 0) in BF16 than in FP64 are left out with their neighbours: those
whose phi0 lies within 0.02 of 0 (BF16 keeps phi to 2^-9 of 0.45, and six steps
move it by less than the rest).  Bound: that of a BF16 state, as in
test_gpu_adjoint_march.py."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import Oracle
from test_gpu_adjoint_march import BOUNDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(32, 8, 3), (96, 24, 7), (64, 16, 40)])
def test_bf16_window_gradient_away_from_the_interface(lib, shape):
    from lbm_bench_gpu_gb300 import capi
    nx, ny, nz = shape
    kw = dict(rhoL=0.1, rhoH=1.0, tauRho=0.7, tauPhi=1.0, width=4.0, sigma=1e-3, Gamma=1.0)
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    s = np.cos(2 * np.pi * x / nx + 0.3) + np.cos(2 * np.pi * y / ny - 0.8) + np.cos(2 * np.pi * z / nz + 1.1)
    phi0 = (0.45 * np.tanh(1.5 * (s - 0.4))).astype(np.float32)
    rho0 = np.full(phi0.shape, 0.55, np.float32)
    T, window, grav = 6, 4, -1e-3
    o = Oracle(nx, ny, nz, **kw)
    o.init(phi0.astype(np.float64), rho0.astype(np.float64))
    _, _, lf, lg = o.adjoint(T, grav, "light_uz_mean", window)
    lphi, _ = o.init_adjoint(phi0.astype(np.float64), lf, lg)
    p = capi.make_params(nx, ny, nz, storage="bf16", **kw)
    with capi.Lattice.from_fields(p, phi0, rho0) as lat:
        r = lat.adjoint(T, grav, "light_uz_mean", window, checkpoint_bytes=3.5 * phi0.size * 54)
    near = np.abs(phi0) < 0.02
    out = near.copy()
    for axis in range(3):
        for d in (-1, 1):
            out |= np.roll(near, d, axis)
    assert out.mean() < 0.5
    assert np.abs(r["dJ_dphi0"] - lphi)[~out].max() <= BOUNDS["bf16"][2] * np.abs(lphi).max()
