"""lbm_stats_noalloc (the statistics kernel) on boxes of every remainder of its
tiles and plane runs, against the same sums in FP64 numpy, and with non-finite
nodes."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PHYS = dict(rhoL=0.1, rhoH=1.0, tauRho=0.7, tauPhi=1.0, width=4.0, sigma=1e-3, Gamma=1.0)


def _raw(lib, p, fields):
    import torch
    from lbm_bench_gpu_gb300 import capi
    dev = [torch.from_numpy(f).cuda() for f in fields]
    out = torch.full((16,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = lib.lbm_stats_noalloc(C.byref(p), *[C.c_void_p(d.data_ptr()) for d in dev], C.c_void_p(out.data_ptr()), None)
    assert rc == capi.LBM_OK
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _want(p, fields):
    from lbm_bench_gpu_gb300 import capi
    d = capi.derive(p)
    good = np.isfinite(np.stack(fields)).all(axis=0)
    phi, rho, ux, uy, uz = [np.where(good, f, 0.0).astype(np.float64) for f in fields]

    def at(dx, dy, dz):   # phi(x + d)
        return np.roll(phi, (-dz, -dy, -dx), (0, 1, 2))

    lap, g = -24.0 * phi, [0.0, 0.0, 0.0]
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                if abs(dx) + abs(dy) + abs(dz) in (1, 2):
                    v = at(dx, dy, dz) * (2.0 if abs(dx) + abs(dy) + abs(dz) == 1 else 1.0)
                    lap = lap + v
                    for k, c in enumerate((dx, dy, dz)):
                        g[k] = g[k] + c * v
    lap, g = lap / 6.0, [v / 12.0 for v in g]
    star = float(d.phiStarSq)
    pres = float(d.alpha) * (phi**2 * (3 * phi**2 - 2 * star) - star**2) \
        - float(d.kappa) * (phi * lap - 0.5 * sum(v * v for v in g)) + rho / 3.0
    u2 = ux**2 + uy**2 + uz**2
    region = good.copy()
    region[:, 0], region[:, -1], region[:, :, 0], region[:, :, -1] = False, False, False, False
    heavy, light = region & (phi >= 0), region & (phi < 0)
    sums = [(u2 * region).max(), heavy.sum(), *[(v * heavy).sum() for v in (ux, uy, uz)], (pres * heavy).sum(),
            (pres * light).sum(), phi.sum(), rho.sum(), *[(rho * v).sum() for v in (ux, uy, uz)],
            (good & (phi >= 0)).sum(), u2.max(), (~good).sum(), 0.0]
    # a sum's bound: the pressure is evaluated in float per node (at most 16 roundings of terms no larger than
    # max|p| + kappa * 24 max phi^2), |u|^2 in 5; the others are sums of ~48 bits of exact terms
    node = np.abs(pres).max() + float(d.kappa) * 48.0 * np.abs(phi).max() ** 2
    eps, n = 2.0**-24, phi.size
    tol = np.array([6 * eps * u2.max(), 0] + [2.0**-40 * np.abs(v).sum() for v in (ux, uy, uz)]
                   + [16 * eps * node * n] * 2 + [2.0**-40 * np.abs(v).sum() for v in (phi, rho)]
                   + [2.0**-40 * np.abs(rho * v).sum() for v in (ux, uy, uz)] + [0, 6 * eps * u2.max(), 0, 0])
    return np.array(sums, np.float64), tol


def _fields(shape, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = shape
    phi = (0.45 * np.tanh(rng.normal(size=(nz, ny, nx)))).astype(np.float32)
    rho = (0.55 + 1e-2 * rng.normal(size=phi.shape)).astype(np.float32)
    return [phi, rho] + [(1e-3 * rng.normal(size=phi.shape)).astype(np.float32) for _ in range(3)]


@pytest.mark.parametrize("shape", [(3, 3, 3), (32, 8, 3), (31, 7, 4), (33, 9, 5), (65, 17, 18), (64, 16, 33),
                                   (150, 90, 71), (300, 41, 130)])
def test_statistics_on_ragged_boxes(lib, shape):
    from lbm_bench_gpu_gb300 import capi
    p = capi.make_params(*shape, **PHYS)
    fields = _fields(shape, 7)
    got = _raw(lib, p, fields)
    want, tol = _want(p, fields)
    assert np.all(np.abs(got - want) <= tol), (got, want, tol)


def test_non_finite_nodes_are_counted_and_left_out(lib):
    from lbm_bench_gpu_gb300 import capi
    shape = (45, 19, 11)
    p = capi.make_params(*shape, **PHYS)
    fields = _fields(shape, 8)
    # non-finite u and rho only: a non-finite phi also enters its neighbours' pressure
    fields[2][3, 4, 5], fields[1][10, 18, 44], fields[4][5, 9, 0], fields[3][7, 7, 7] = np.nan, np.inf, -np.inf, np.nan
    got = _raw(lib, p, fields)
    want, tol = _want(p, fields)
    # the left-out nodes keep their phi in their neighbours' stencils: at most 7 nodes' surface terms each
    d = capi.derive(p)
    tol[5:7] += 4 * 19 * float(d.kappa) * 48.0 * 0.45**2
    assert got[14] == 4
    assert np.all(np.abs(got - want) <= tol), (got, want, tol)
