"""The workloads whose speed is tracked, as a program that uses the library runs them.

A case is a dict of plain values; ``kind`` says which calls one pass makes:

  step     a lattice that is being evolved: ``steps`` fused steps, then the point at which a
           driver looks at the run (lbm_stats with the phi, rho and u fields copied into its own
           pinned host buffers), all through one context that a pass leaves further on
  run      a short run from the bubble list to the fields: lbm_init_bubbles, ``steps`` steps,
           lbm_stats with the fields, lbm_destroy
  monitor  in-situ statistics of fields that another program keeps on the GPU (lbm_stats_noalloc)
  adjoint  J, dJ/d(body force) and dJ/dphi0 over ``steps`` steps with ``slots`` checkpoints
           (lbm_step_adjoint)

Boxes, bubble radii and densities, relaxation times and the body force are those of the
workloads in ``lbm_bench_gpu_gb300/inputs.py``, of the tests and of ``bench.py``.  ``exact``
restates the step, its transpose (by automatic differentiation) and the statistics in 64-bit
torch; it uses none of the library's code.
"""
import ctypes
import math

import numpy as np
import torch

from lbm_bench_gpu_gb300 import capi
from lbm_bench_gpu_gb300.inputs import place_bubbles

FIELDS = ("phi", "rho", "ux", "uy", "uz")
PHYSICS = {"rhoL": 0.1, "rhoH": 1.0, "tauPhi": 1.0, "width": 4.0, "sigma": 1e-3, "Gamma": 1.0}
ELEMENT = {"fp32": 4, "fp16": 2, "bf16": 2}


def _box(nx, ny, nz, **more):
    return {"nx": nx, "ny": ny, "nz": nz, **more}


def listed():
    return [
        # the smallest box the tests step, looked at after a few steps: launches and latency
        {"name": "step_fp32_32", "kind": "step", **_box(32, 32, 32), "storage": "fp32", "steps": 10, "grav": -1e-6},
        # the static bubble of the Laplace check (relaxation without gravity)
        {"name": "static_fp32_64", "kind": "step", **_box(64, 64, 64), "storage": "fp32", "steps": 100, "grav": 0.0},
        # an ordinary box that half fills the chip
        {"name": "step_fp32_128", "kind": "step", **_box(128, 128, 128), "storage": "fp32", "steps": 50,
         "grav": -1e-6},
        # a box with no equal or round sides, in the third storage format
        {"name": "step_bf16_ragged", "kind": "step", **_box(160, 104, 93), "storage": "bf16", "steps": 50,
         "grav": -1e-6},
        # the benchmark's bubbly flow, in its own format and in the 16-bit one
        {"name": "step_fp32_256", "kind": "step", **_box(256, 256, 256), "storage": "fp32", "steps": 50,
         "grav": -1e-6},
        {"name": "step_fp16_256", "kind": "step", **_box(256, 256, 256), "storage": "fp16", "steps": 50,
         "grav": -1e-6},
        # the largest bubbly flow
        {"name": "step_fp16_512", "kind": "step", **_box(512, 512, 512), "storage": "fp16", "steps": 20,
         "grav": -1e-6},
        # a short run of a parameter study, from the bubble list to the fields
        {"name": "run_fp16_192", "kind": "run", **_box(192, 192, 192), "storage": "fp16", "steps": 20,
         "grav": -1e-6},
        # a monitoring hook of another program, on the benchmark's box
        {"name": "monitor_256", "kind": "monitor", **_box(256, 256, 256)},
        # gradients at the size of the finite-difference checks
        {"name": "adjoint_fp32_64", "kind": "adjoint", **_box(64, 64, 64), "storage": "fp32", "steps": 60,
         "objective": "light_z_centroid", "window": 1, "slots": 12, "grav": -1e-6},
        # the short adjoint workload: recomputation, an averaging window
        {"name": "adjoint_fp32_128", "kind": "adjoint", **_box(128, 128, 128), "storage": "fp32", "steps": 60,
         "objective": "light_uz_mean", "window": 12, "slots": 12, "grav": -1e-6},
        # the long-horizon workload's box and format, few checkpoints for its steps
        {"name": "adjoint_fp16_256", "kind": "adjoint", **_box(256, 256, 256), "storage": "fp16", "steps": 16,
         "objective": "light_z_centroid", "window": 1, "slots": 6, "grav": -1e-6},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "run", "monitor", "adjoint", "adjoint"])
    if kind == "monitor":   # any sides from 3 up
        return {"kind": kind, **_box(*(_log_int(rng, 16, 300) for _ in range(3)))}
    top = 128 if kind == "adjoint" else 256
    box = _box(32 * _log_int(rng, 1, top // 32), 8 * _log_int(rng, 4, top // 8), _log_int(rng, 26, top))
    case = {"kind": kind, **box, "storage": rng.choice(["fp32", "fp16", "bf16"]),
            "grav": rng.choice([0.0, -1e-6, -1e-6])}
    if kind == "step":
        case["steps"] = _log_int(rng, 10, 100)
    elif kind == "run":
        case["steps"] = _log_int(rng, 10, 40)
    else:
        case["steps"] = _log_int(rng, 8, 60)
        case["objective"] = rng.choice(["light_uz_mean", "light_z_centroid"])
        case["window"] = rng.randint(1, case["steps"]) if case["objective"] == "light_uz_mean" else 1
        case["slots"] = rng.randint(4, 24)
        case["grav"] = -1e-6
    return case


# ---- inputs ----

def _bubbles(case, seed):
    """One bubble for each 64^3 of the box, as in the benchmark; radii smaller where a side is short."""
    box = (case["nx"], case["ny"], case["nz"])
    most = min(10.0, min(box) / 2 - 7.0)
    count = max(1, round(box[0] * box[1] * box[2] / 64**3))
    for n in range(count, 0, -1):
        try:
            return place_bubbles(n, box, (min(6.0, 0.7 * most), most), seed=seed, max_tries=40 * n + 1000)
        except RuntimeError:   # no room for that many in a thin box
            pass
    raise ValueError("no bubble fits the box")


def _tau_rho(case):
    return 0.8 if case["kind"] == "adjoint" else 0.7


def _params(case, bubbles):
    return capi.make_params(case["nx"], case["ny"], case["nz"], tauRho=_tau_rho(case), rc0=float(bubbles[0, 3]),
                            storage=case["storage"], **PHYSICS)


def _host_fields(case):
    """The program's own pinned buffers for phi, rho, u (written once, so that their pages are there)."""
    shape = (case["nz"], case["ny"], case["nx"])
    return {k: torch.zeros(shape, dtype=torch.float32, pin_memory=True).numpy() for k in FIELDS}


def _monitor_fields(case, seed):
    """phi of a few bubbles, density and velocity of a slow flow around them, on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dev = {"device": "cuda", "dtype": torch.float32}
    z, y, x = torch.meshgrid(torch.arange(nz, **dev), torch.arange(ny, **dev), torch.arange(nx, **dev), indexing="ij")
    star = 0.5 * (PHYSICS["rhoH"] - PHYSICS["rhoL"])
    phi = torch.full((nz, ny, nx), -star, **dev)
    where = torch.rand(6, 4, generator=gen, **dev).cpu().tolist()
    for a, b, c, r in where:
        dist = torch.sqrt((x - a * nx) ** 2 + (y - b * ny) ** 2 + (z - c * nz) ** 2)
        phi = torch.maximum(phi, star * torch.tanh(2 * (6 + 6 * r - dist) / PHYSICS["width"]))
    rho = 0.55 + 1e-3 * torch.randn(phi.shape, generator=gen, **dev)
    u = [1e-4 * torch.randn(phi.shape, generator=gen, **dev) + 5e-5 * (k == 2) * phi for k in range(3)]
    return [phi.contiguous(), rho, *[v.contiguous() for v in u]]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "monitor":
        # rhoL and the others only enter the pressure's constants
        p = capi.make_params(case["nx"], case["ny"], case["nz"], tauRho=0.7, **PHYSICS)
        return {"kind": kind, "params": p, "fields": _monitor_fields(case, seed),
                "raw": torch.zeros(16, dtype=torch.float64, device="cuda")}
    bubbles = _bubbles(case, seed)
    state = {"kind": kind, "case": dict(case), "params": _params(case, bubbles), "bubbles": bubbles}
    if kind in ("step", "run"):
        state["host"] = _host_fields(case)
    if kind in ("step", "adjoint"):
        state["lattice"] = capi.Lattice.from_bubbles(state["params"], bubbles)
    return state


# ---- one pass ----

def _look(lat, host):
    """lbm_stats with the fields copied into the program's buffers."""
    s = capi.StatsOut()
    capi.check(capi.load().lbm_stats(lat._h, ctypes.byref(s), *[capi.fptr(host[k]) for k in FIELDS]), "lbm_stats")
    return {"fields": host, "stats": s.as_dict()}


def _snapshot_bytes(case):
    n = case["nx"] * case["ny"] * case["nz"]
    return n * (4 + 25 * ELEMENT[case["storage"]])


def run(state):
    if state["kind"] == "monitor":
        stream = torch.cuda.current_stream().cuda_stream
        code = capi.load().lbm_stats_noalloc(ctypes.byref(state["params"]), *[f.data_ptr() for f in state["fields"]],
                                             state["raw"].data_ptr(), stream)
        capi.check(code, "lbm_stats_noalloc")
        return state["raw"]
    case = state["case"]
    if state["kind"] == "step":
        state["lattice"].step(case["steps"], case["grav"])
        return _look(state["lattice"], state["host"])
    if state["kind"] == "run":
        with capi.Lattice.from_bubbles(state["params"], state["bubbles"]) as lat:
            lat.step(case["steps"], case["grav"])
            return _look(lat, state["host"])
    r = state["lattice"].adjoint(case["steps"], case["grav"], case["objective"], case["window"],
                                 checkpoint_bytes=(case["slots"] + 0.5) * _snapshot_bytes(case))
    return {k: r[k] for k in ("J", "dJ_dgrav", "dJ_dphi0")}


def work(case):
    """Each step reads and writes its 26 distributions once (f_0 always FP32); an adjoint step reads
    the adjoint distributions and the state and writes the adjoint distributions once; a forward
    trajectory is needed once, however often checkpoints make it be recomputed."""
    n = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "monitor":
        return {"bytes": 20 * n + 128, "flops": 90 * n}
    state = 4 + 25 * ELEMENT[case["storage"]]
    steps = case["steps"]
    if case["kind"] == "adjoint":
        return {"bytes": n * (steps * (2 * state + 2 * 104 + state) + 4), "flops": n * steps * (420 + 700)}
    read_back = 20 * 2 * n   # the five fields, written by the last step and read for the statistics and the copy
    return {"bytes": n * steps * 2 * state + read_back, "flops": 420 * n * steps}


# ---- the same in 64 bits ----

C7 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]
C19 = C7 + [(1, 1, 0), (-1, -1, 0), (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1),
            (0, 1, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1)]
W19 = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12


def _constants(tau_rho):
    k = {name: float(np.float32(v)) for name, v in PHYSICS.items()}
    star = 0.5 * (k["rhoH"] - k["rhoL"])
    tr = float(np.float32(tau_rho))
    alpha = 0.75 * k["sigma"] / (k["width"] * star**4)
    eta = 1.0 / (k["tauPhi"] + 0.5)
    return {"star": star, "alpha": alpha, "kappa": 0.5 * alpha * (k["width"] * star) ** 2, "eta": eta,
            "width": k["width"], "Gamma": k["Gamma"], "tr": tr, "tp": k["tauPhi"], "rho0": 0.5 * (k["rhoH"] + k["rhoL"])}


def _at(a, c):
    """a(x + c), periodic."""
    return torch.roll(a, (-c[2], -c[1], -c[0]), (0, 1, 2))


def _stencils(phi):
    """Laplacian and gradient on the 19 points (faces weigh twice the edges)."""
    lap = -24.0 * phi
    grad = [0.0, 0.0, 0.0]
    for i in range(1, 19):
        v = _at(phi, C19[i]) * (2.0 if i < 7 else 1.0)
        lap = lap + v
        for d in range(3):
            if C19[i][d]:
                grad[d] = grad[d] + C19[i][d] * v
    return lap / 6.0, [g / 12.0 for g in grad]


def _mu(phi, lap, k):
    return 4.0 * k["alpha"] * phi * (phi * phi - k["star"] ** 2) - k["kappa"] * lap


def _bubble_phi(case, bubbles, k):
    """phi of the bubble list; which nodes a bubble covers is decided in 32 bits, as its inputs are."""
    dev = {"device": "cuda"}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    z, y, x = torch.meshgrid(torch.arange(1, nz + 1, **dev), torch.arange(ny, **dev), torch.arange(nx, **dev),
                             indexing="ij")
    phi = torch.full((nz, ny, nx), -k["star"], dtype=torch.float64, **dev)
    for xc, yc, zc, rc in np.asarray(bubbles, np.float32):
        d = [(a.float() - float(b)) for a, b in ((x, xc), (y, yc), (z, zc))]
        inside = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]) <= float(np.float32(rc + np.float32(k["width"])))
        r = torch.sqrt(sum((a.double() - float(b)) ** 2 for a, b in ((x, xc), (y, yc), (z, zc))))
        phi = torch.where(inside, k["star"] * torch.tanh(2.0 * (float(rc) - r) / k["width"]), phi)
    return phi


def _initial(phi, k):
    mu = _mu(phi, _stencils(phi)[0], k)
    f = [phi - 3.0 * k["Gamma"] * mu] + [0.5 * k["Gamma"] * mu] * 6
    g = [k["rho0"] / 3.0 - 2.0 * phi * mu] + [w * (3.0 * phi * mu + k["rho0"]) for w in W19[1:]]
    return f + g


def _moments(s):
    phi, rho = sum(s[1:7], s[0]), sum(s[8:], s[7])
    u = []
    for d in range(3):
        m = 0.0
        for i in range(1, 19):
            if C19[i][d]:
                m = m + C19[i][d] * s[7 + i]
        u.append(m / rho)
    return phi, rho, u


def _step(s, k, grav):
    phi, rho, u = _moments(s)
    lap, grad = _stencils(phi)
    mu = _mu(phi, lap, k)
    force = [mu * g for g in grad]
    force[2] = force[2] + grav * (phi > 0).double()
    us = [a + 0.5 * b / rho for a, b in zip(u, force)]
    uf = us[0] * force[0] + us[1] * force[1] + us[2] * force[2]
    v = [3.0 * a for a in us]
    vsq = (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) / 6.0
    new = []
    a, cf, af = 1.0 - 1.0 / k["tp"], phi * (0.5 / (1.0 - k["eta"])) / k["tp"], 0.5 * k["Gamma"] / k["tp"] * mu
    for i in range(7):
        if i == 0:
            post = a * s[0] - 6.0 * af + phi / k["tp"]
        else:
            d = (i - 1) // 2
            post = a * s[i] + af + C7[i][d] * cf * us[d]
        new.append(post if i == 0 else k["eta"] * _at(post, tuple(-c for c in C7[i])) + (1.0 - k["eta"]) * post)
    b, inv = 1.0 - 1.0 / k["tr"], 1.0 / k["tr"]
    half = 1.0 - 0.5 * inv
    iso = 3.0 * phi * mu + rho * (1.0 - vsq)
    for i in range(19):
        if i == 0:
            post = b * s[7] + inv / 3.0 * (rho - 6.0 * phi * mu - rho * vsq) - half * uf
        else:
            c = C19[i]
            w, wf = 0.0, 0.0
            for d in range(3):
                if c[d]:
                    w, wf = w + c[d] * v[d], wf + c[d] * force[d]
            kw, kc = (inv / 18.0, half / 6.0) if i < 7 else (inv / 36.0, half / 12.0)
            # the odd part of the forcing is w (c.F) on the axes and c.F on the diagonals (src/collision_g.cu:111-196)
            post = (b * s[7 + i] + kw * iso + 0.5 * kw * rho * w * w + kc * (w * wf - uf) + kw * rho * w
                    + (kc * w * wf * _sign(c) if i < 7 else kc * wf))
        new.append(_at(post, tuple(-q for q in C19[i])))
    return new


def _sign(c):
    return float(sum(c))


def _exact_fields(case, seed):
    k = _constants(_tau_rho(case))
    grav = float(np.float32(case["grav"]))
    with torch.no_grad():
        s = _initial(_bubble_phi(case, _bubbles(case, seed), k), k)
        for _ in range(case["steps"] - 1):   # the fields are the moments at the start of the last step
            s = _step(s, k, grav)
        phi, rho, u = _moments(s)
    return {"fields": dict(zip(FIELDS, (phi, rho, *u))), "stats": None}


def _weighted(case, s, k):
    """The light phase's mean of u_z or of the plane number."""
    phi, _, u = _moments(s)
    w = (k["star"] - phi) / (2.0 * k["star"])
    q = u[2] if case["objective"] == "light_uz_mean" else \
        torch.arange(1, case["nz"] + 1, device="cuda", dtype=torch.float64)[:, None, None]
    return (w * q).sum() / w.sum()


def _exact_adjoint(case, seed):
    k = _constants(_tau_rho(case))
    grav = torch.tensor(float(np.float32(case["grav"])), dtype=torch.float64, device="cuda", requires_grad=True)
    steps, window = case["steps"], case["window"]
    first = steps - window + 1 if case["objective"] == "light_uz_mean" else steps
    phi0 = _bubble_phi(case, _bubbles(case, seed), k).requires_grad_()
    with torch.no_grad():
        states = [_initial(phi0, k)]
        for _ in range(steps):
            states.append(_step(states[-1], k, grav))
    total, d_grav = 0.0, 0.0
    lam = [torch.zeros_like(phi0) for _ in range(26)]
    for n in range(steps, -1, -1):
        s = [a.detach().requires_grad_() for a in states[n]]
        states[n] = None
        if n >= first:
            j = _weighted(case, s, k) / window
            total += float(j.detach())
            got = torch.autograd.grad(j, s, allow_unused=True)
            lam = [a if b is None else a + b for a, b in zip(lam, got)]
        if n == 0:
            break
        prev = [a.detach().requires_grad_() for a in states[n - 1]]
        got = torch.autograd.grad(_step(prev, k, grav), [grav] + prev, lam)
        d_grav += float(got[0])
        lam = list(got[1:])
    (d_phi,) = torch.autograd.grad(_initial(phi0, k), [phi0], lam)
    return {"J": total, "dJ_dgrav": d_grav, "dJ_dphi0": d_phi}


def _exact_monitor(case, seed):
    k = _constants(0.7)
    phi, rho, *u = [a.double() for a in _monitor_fields(case, seed)]
    u2 = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
    lap, grad = _stencils(phi)
    sq = phi * phi
    pressure = (k["alpha"] * (sq * (3.0 * sq - 2.0 * k["star"] ** 2) - k["star"] ** 4)
                - k["kappa"] * (phi * lap - 0.5 * (grad[0] ** 2 + grad[1] ** 2 + grad[2] ** 2)) + rho / 3.0)
    inner = (slice(None), slice(1, -1), slice(1, -1))   # the region the reference's statistics cover
    heavy = phi[inner] >= 0
    raw = [u2[inner].max(), heavy.sum(), *[(a[inner] * heavy).sum() for a in u], (pressure[inner] * heavy).sum(),
           (pressure[inner] * ~heavy).sum(), phi.sum(), rho.sum(), *[(rho * a).sum() for a in u], (phi >= 0).sum(),
           u2.max(), torch.zeros(()), torch.zeros(())]
    return torch.stack([v.double().cuda() for v in raw])


def exact(case, seed):
    n = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "monitor":
        return _exact_monitor(case, seed)
    if n * case["steps"] > 1.2e9:   # 64-bit steps of the largest box take longer than they are worth
        return None
    return _exact_adjoint(case, seed) if case["kind"] == "adjoint" else _exact_fields(case, seed)
