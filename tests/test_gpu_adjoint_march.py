"""The adjoint's z-marching kernel against the oracle's FP64 adjoint where its
tiles end: one tile in x (both periodic seams in one tile, also of the 16-bit
pair layout), one tile in y, few planes, several plane runs; with the seven
lambda_f fields merged into one (tauPhi = 1) and kept apart.  An interface
crosses every seam.  Bounds (J, dJ/dgrav, dJ/dphi0 of its max) as in
test_gpu_adjoint.py."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

BOUNDS = {"fp32": (1e-5, 1e-3, 2e-3), "fp16": (1e-4, 1e-3, 1e-3), "bf16": (1e-3, 1e-2, 1e-2)}


@pytest.mark.parametrize("storage", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("shape,tau_phi", [((32, 8, 3), 1.0), ((32, 16, 5), 0.8), ((64, 8, 9), 1.0),
                                           ((96, 24, 7), 1.0), ((64, 32, 70), 1.0), ((96, 16, 11), 1.2)])
def test_gradient_matches_oracle(lib, storage, shape, tau_phi):
    from lbm_bench_gpu_gb300 import capi
    nx, ny, nz = shape
    kw = dict(rhoL=0.1, rhoH=1.0, tauRho=0.7, tauPhi=tau_phi, width=4.0, sigma=1e-3, Gamma=1.0)
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    s = np.cos(2 * np.pi * x / nx + 0.3) + np.cos(2 * np.pi * y / ny - 0.8) + np.cos(2 * np.pi * z / nz + 1.1)
    phi0 = (0.45 * np.tanh(1.5 * (s - 0.4))).astype(np.float32)
    rho0 = np.full(phi0.shape, 0.55, np.float32)
    T, grav = 5, -3e-5
    p = capi.make_params(nx, ny, nz, storage=storage, **kw)
    o = Oracle(nx, ny, nz, **kw)
    o.init(phi0.astype(np.float64), rho0.astype(np.float64))
    J, dg, lf, lg = o.adjoint(T, grav, "light_z_centroid", 1)
    lphi, _ = o.init_adjoint(phi0.astype(np.float64), lf, lg)
    snap = phi0.size * (104 if storage == "fp32" else 54)
    with capi.Lattice.from_fields(p, phi0, rho0) as lat:
        r = lat.adjoint(T, grav, "light_z_centroid", 1, checkpoint_bytes=3.5 * snap)
    bj, bg, bp = BOUNDS[storage]
    assert r["J"] == pytest.approx(J, rel=bj)
    assert r["dJ_dgrav"] == pytest.approx(dg, rel=bg)
    assert np.abs(r["dJ_dphi0"] - lphi).max() <= bp * np.abs(lphi).max()


# The window steps of the u_z objective take their sums from the phi kernel
# (weights) and the march kernel (w u_z).  Against lbm_objective, whose sums come
# from one pass over the states: the same float terms in FP64 sums of another
# order, n 2^-53 apart at most (5e-12 for the largest box here; gravity gives the
# terms one sign, so J does not cancel).  The gradient as above for FP32 and
# FP16; with a BF16 state a node at phi0 = -0.0035 crosses into the heavy set,
# which puts its entry 1.3 % from the FP64 one whatever kernel computes it.
@pytest.mark.parametrize("storage", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("shape", [(32, 8, 3), (96, 24, 7), (64, 16, 40)])
def test_window_sums_and_gradient(lib, storage, shape):
    from lbm_bench_gpu_gb300 import capi
    nx, ny, nz = shape
    kw = dict(rhoL=0.1, rhoH=1.0, tauRho=0.7, tauPhi=1.0, width=4.0, sigma=1e-3, Gamma=1.0)
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    s = np.cos(2 * np.pi * x / nx + 0.3) + np.cos(2 * np.pi * y / ny - 0.8) + np.cos(2 * np.pi * z / nz + 1.1)
    phi0 = (0.45 * np.tanh(1.5 * (s - 0.4))).astype(np.float32)
    rho0 = np.full(phi0.shape, 0.55, np.float32)
    T, window, grav = 6, 4, -1e-3
    p = capi.make_params(nx, ny, nz, storage=storage, **kw)
    o = Oracle(nx, ny, nz, **kw)
    o.init(phi0.astype(np.float64), rho0.astype(np.float64))
    _, dg, lf, lg = o.adjoint(T, grav, "light_uz_mean", window)
    lphi, _ = o.init_adjoint(phi0.astype(np.float64), lf, lg)
    snap = phi0.size * (104 if storage == "fp32" else 54)
    with capi.Lattice.from_fields(p, phi0, rho0) as lat:
        r = lat.adjoint(T, grav, "light_uz_mean", window, checkpoint_bytes=3.5 * snap)
        J = lat.objective(T, grav, "light_uz_mean", window)
    _, bg, bp = BOUNDS[storage]
    assert r["J"] == pytest.approx(J, rel=1e-9)
    assert r["dJ_dgrav"] == pytest.approx(dg, rel=bg)
    if storage != "bf16":
        assert np.abs(r["dJ_dphi0"] - lphi).max() <= bp * np.abs(lphi).max()
