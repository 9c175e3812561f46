"""Boxes longer in y or z than a CUDA grid's second and third dimension allow
tiles (65535 of them): lbm_init, steps and statistics accept every box the
parameter checks accept.  The initial fields repeat along the long side with the
length of a small box, so every repetition evolves like that box, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KW = dict(rhoL=0.1, rhoH=1.0, tauRho=0.7, tauPhi=1.0, width=4.0, sigma=1e-3, Gamma=1.0)


@pytest.mark.parametrize("storage", ["fp32", "fp16"])
@pytest.mark.parametrize("shape,small", [((32, 8 * 65537, 3), (32, 8, 3)), ((32, 8, 4 * 65537), (32, 8, 4))])
def test_long_box_evolves_like_its_repeated_part(lib, storage, shape, small):
    from lbm_bench_gpu_gb300 import capi
    rng = np.random.default_rng(5)
    nx, ny, nz = small
    phi = (0.45 * np.tanh(rng.normal(size=(nz, ny, nx)))).astype(np.float32)
    rho = np.full(phi.shape, 0.55, np.float32)
    reps = (shape[2] // nz, shape[1] // ny, 1)

    def run(box, a, b):
        p = capi.make_params(*box, storage=storage, **KW)
        with capi.Lattice.from_fields(p, a, b) as lat:
            lat.step(2, -1e-5)
            return lat.fields()

    want = run(small, phi, rho)
    got = run(shape, np.tile(phi, reps), np.tile(rho, reps))
    for k, v in want.items():
        parts = got[k].reshape(reps[0], nz, reps[1], ny, nx)
        assert np.array_equal(parts, np.broadcast_to(v[None, :, None], parts.shape)), k
