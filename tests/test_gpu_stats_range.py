"""The statistics' sums in FP64 from each thread's own sum on: a sum over many
nodes may leave the range of FP32 (its nodes' values do not), and keeps FP64
accuracy across threads.  A node left out for its u or rho still counts in its
neighbours' pressure."""
from __future__ import annotations

import math

import numpy as np
import pytest

from test_gpu_stats_sizes import PHYS, _fields, _raw, _want

pytestmark = pytest.mark.gpu


# Boxes of at most two nodes a thread: 3e38 there is within FP32.  Each sum is
# one of equal terms with at most 24 bits, exact up to the roundings of FP64.
@pytest.mark.parametrize("shape", [(3, 3, 3), (32, 16, 4), (33, 9, 5), (64, 33, 7)])
def test_sums_beyond_fp32(lib, shape):
    from lbm_bench_gpu_gb300 import capi
    p = capi.make_params(*shape, **PHYS)
    nx, ny, nz = shape
    n, big = nx * ny * nz, np.float32(1.5e38)
    phi = np.full((nz, ny, nx), -0.45, np.float32)
    rho = np.full(phi.shape, big)
    u = [np.full(phi.shape, np.float32(v)) for v in (1.0, -0.5, 0.25)]
    got = _raw(lib, p, [phi, rho] + u)
    want = np.array([float(big) * n, float(big) * n, -0.5 * float(big) * n, 0.25 * float(big) * n])
    assert np.all(np.abs(got[8:12] - want) <= n * 2.0**-53 * np.abs(want)), (got[8:12], want)
    # all of the region is light: p = rho / 3 (and terms of phi below its rounding), in FP32 a node
    region = (nx - 2) * (ny - 2) * nz
    assert got[6] == pytest.approx(region * float(big) / 3.0, rel=2.0**-22)
    assert got[14] == 0


# A warp whose threads' sums all reach the top of FP32's range.
def test_sums_at_the_end_of_fp32(lib):
    from lbm_bench_gpu_gb300 import capi
    shape = (64, 32, 4)
    p = capi.make_params(*shape, **PHYS)
    nx, ny, nz = shape
    n, big = nx * ny * nz, np.float32(2.0**127 * (1 - 2.0**-24))   # two of them: FP32's largest value
    phi = np.full((nz, ny, nx), -0.45, np.float32)
    rho = np.full(phi.shape, big)
    u = [np.full(phi.shape, np.float32(v)) for v in (1.0, -0.5, 0.25)]
    got = _raw(lib, p, [phi, rho] + u)
    want = float(big) * n
    assert abs(got[8] - want) <= n * 2.0**-53 * want and abs(got[9] - want) <= n * 2.0**-53 * want


def test_pressure_beside_left_out_nodes(lib):
    from lbm_bench_gpu_gb300 import capi
    shape = (45, 19, 11)
    p = capi.make_params(*shape, **PHYS)
    fields = _fields(shape, 8)
    clean = [f.copy() for f in fields]
    bad = [(2, (3, 4, 5)), (1, (10, 18, 44)), (4, (5, 9, 0)), (3, (7, 7, 7)), (3, (4, 10, 20)), (1, (0, 5, 9))]
    for f, at in bad:
        fields[f][at] = math.nan
    got = _raw(lib, p, fields)
    # the whole box's pressure sums less those of the left-out nodes, each summed alone in FP64
    whole, tol = _want(p, clean)
    assert got[14] == len(bad)
    left = {5: 0.0, 6: 0.0}
    for _, at in bad:
        z, y, x = at
        if not (1 <= y <= shape[1] - 2 and 1 <= x <= shape[0] - 2):
            continue
        heavy = clean[0][at] >= 0
        left[5 if heavy else 6] += _node_pressure(p, clean, at)
    for v in (5, 6):
        assert abs(got[v] - (whole[v] - left[v])) <= tol[v], (v, got[v], whole[v] - left[v], tol[v])


def _node_pressure(p, fields, at):
    """p of one node (src/logsave.c:94-137) in FP64, periodic."""
    from lbm_bench_gpu_gb300 import capi
    d = capi.derive(p)
    phi, rho = fields[0].astype(np.float64), float(fields[1][at])
    c, lap, g = phi[at], -24.0 * phi[at], np.zeros(3)
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                k = abs(dx) + abs(dy) + abs(dz)
                if k in (1, 2):
                    v = phi[tuple((i + s) % m for i, s, m in zip(at, (dz, dy, dx), phi.shape))] * (2.0 if k == 1 else 1.0)
                    lap += v
                    g += np.array((dx, dy, dz)) * v
    lap, g = lap / 6.0, g / 12.0
    star = float(d.phiStarSq)
    return float(d.alpha) * (c**2 * (3 * c**2 - 2 * star) - star**2) - float(d.kappa) * (c * lap - 0.5 * g @ g) + rho / 3.0


# Boxes of few rows: a block's warps share its tile's rows and several runs of planes.
@pytest.mark.parametrize("shape", [(70, 3, 50), (40, 4, 37), (33, 5, 19), (64, 8, 70), (5, 6, 333), (65, 8, 3),
                                   (32, 3, 3), (700, 4, 1100)])
def test_statistics_of_thin_boxes(lib, shape):
    from lbm_bench_gpu_gb300 import capi
    p = capi.make_params(*shape, **PHYS)
    fields = _fields(shape, 9)
    got = _raw(lib, p, fields)
    want, tol = _want(p, fields)
    assert np.all(np.abs(got - want) <= tol), (got, want, tol)
