"""The work that users of this package have it do, as cases that can be timed and checked.

A case is one pass through a public entry point: a BIA step of a device-resident system
(`BIASolver.step`, in place or on a copy of a state that is kept), a run of steps in one CUDA
graph (`run`), a step of a host state (`run_host`), a run of an ensemble of systems
(`Ensemble.run`), the direct-sum integrator (`dim_integrate`), the conserved quantities
(`invariance`), and a whole step of a host program through the reference's own per-particle
call (`find_dxyuv_kernel` for every particle, then drift and update).  Sizes and physics
are those of the package's workloads (gravity ball of 1332, Coulomb cube and Plummer sphere of
32768, 4096 Plummer systems of 32 to 1024, cold ball of 131072) and ragged sizes between them.

Everything is FP64 (the only type the entry points take); the options are the four methods,
charges, and where the state lives.  The learned form runs with the heads that ship with the
package; training new ones is done once, offline, and is not a case.
"""
import math

import numpy as np
import torch

from bia_3d_gpu_b200 import (METHOD_ALG, METHOD_LEARNED, METHOD_RKF, METHOD_UNIVERSAL, BIASolver, default_config,
                             find_dxyuv_kernel, initial)

METHODS = {"alg": METHOD_ALG, "rkf": METHOD_RKF, "universal": METHOD_UNIVERSAL, "learned": METHOD_LEARNED}


def listed():
    return [
        # a small system stepped from a host loop, one call a step: launch latency
        {"name": "plummer_universal_257", "kind": "step", "workload": "plummer", "method": "universal", "n": 257, "dt": 1e-4},
        # the package's smallest workload as it is run: the reference's algorithm, steps in one graph
        {"name": "ball_alg_1332_run20", "kind": "run", "workload": "ball", "method": "alg", "n": 1332, "dt": 1e-4, "steps": 20},
        # a Fortran-style program that owns the state in host memory, ragged size
        {"name": "plummer_universal_10007_host", "kind": "host", "workload": "plummer", "method": "universal", "n": 10007, "dt": 1e-4},
        # the headline workload: one step of the Plummer sphere, learned form
        {"name": "plummer_learned_32768", "kind": "step", "workload": "plummer", "method": "learned", "n": 32768, "dt": 1e-4},
        # the charged plasma in the reference's algorithm: all orbit classes mixed
        {"name": "coulomb_alg_32768", "kind": "advance", "workload": "coulomb", "method": "alg", "n": 32768, "dt": 1e-5},
        # the same physics in the reference's other mode, adaptive RKF45 per pair, ragged size
        {"name": "coulomb_rkf_8191", "kind": "advance", "workload": "coulomb", "method": "rkf", "n": 8191, "dt": 1e-5},
        # the plasma at a long step, where nearly half the pairs go through the learned heads
        {"name": "coulomb_learned_16384_long", "kind": "advance", "workload": "coulomb", "method": "learned", "n": 16384, "dt": 1e-3},
        # the largest system: cold collapse, every pair radial
        {"name": "cold_learned_131072", "kind": "step", "workload": "cold", "method": "learned", "n": 131072, "dt": 5e-5},
        # thousands of small systems of uneven size advanced together
        {"name": "ensemble_learned_4096", "kind": "ensemble", "method": "learned", "systems": 4096, "nmin": 32, "nmax": 1024, "dt": 1e-4, "steps": 2},
        # the physics check: direct-sum integration over some steps, at the reference run's size
        {"name": "dim_plummer_1332", "kind": "dim", "workload": "plummer", "n": 1332, "t": 5e-3},
        # the reference's driver loop: its drop-in call for every particle, host arrays in and out
        {"name": "rows_alg_1332", "kind": "rows", "workload": "ball", "method": "alg", "n": 1332, "dt": 1e-4},
        # conserved quantities, as taken before and after every run
        {"name": "invariants_32768", "kind": "invariants", "workload": "coulomb", "n": 32768},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step"] * 6 + ["run", "host", "ensemble", "dim", "rows", "invariants"])
    if kind == "ensemble":
        nmax = size(64, 1024)
        return {"kind": kind, "method": rng.choice(["alg", "universal", "learned"]), "systems": size(32, 1024),
                "nmin": rng.randint(16, 32), "nmax": nmax, "dt": 1e-4, "steps": rng.randint(1, 8)}
    if kind == "dim":
        return {"kind": kind, "workload": rng.choice(["plummer", "ball"]), "n": size(200, 6000), "t": size(100, 3000) * 1e-6}
    if kind == "invariants":
        return {"kind": kind, "workload": rng.choice(["plummer", "coulomb", "cold"]), "n": size(200, 65536)}
    if kind == "rows":
        return {"kind": kind, "workload": rng.choice(["plummer", "ball"]), "method": rng.choice(["alg", "alg", "rkf"]),
                "n": size(60, 1400), "dt": 1e-4}
    method = rng.choice(["alg", "rkf", "universal", "learned"])
    workload = rng.choice(["plummer", "coulomb", "ball", "cold"])
    top = {"alg": 20000, "rkf": 12000, "universal": 60000, "learned": 60000}[method]
    dt = {"plummer": 1e-4, "ball": 1e-4, "cold": 5e-5, "coulomb": rng.choice([1e-5, 1e-4]) if method == "learned" else 1e-5}[workload]
    if kind == "step" and workload == "coulomb":
        kind = "advance"
    case = {"kind": kind, "workload": workload, "method": method, "n": size(100, top if kind in ("step", "advance") else 6000), "dt": dt}
    if kind == "run":
        case["steps"] = rng.randint(4, 24)
    return case


# ---- inputs ------------------------------------------------------------------------------


def _system(workload, n, seed):
    """(state (6, n) float64, coupling, charges or None) of one seeded system."""
    if workload == "coulomb":
        return initial.coulomb_cube(n, seed=seed, dmin=min(1e-3, 0.1 * n ** (-1.0 / 3.0)))
    make = {"plummer": initial.plummer, "ball": initial.gravity_ball, "cold": initial.cold_ball}[workload]
    s, eps = make(n=n, seed=seed)
    return s, eps, None


def _sizes(case):
    return initial.ensemble_sizes(case["systems"], case["nmin"], case["nmax"])


def _ensemble(case, seed):
    """(state (6, sum n_s), couplings) of the systems back to back, each a Plummer sphere at rest."""
    sizes = _sizes(case)
    s, _ = initial.plummer(int(sizes.sum()), seed=seed, rmax=20.0)
    first = np.concatenate([[0], np.cumsum(sizes)[:-1]])
    for k in range(6):
        s[k] -= np.repeat(np.add.reduceat(s[k], first) / sizes, sizes)
    return s, -2.0 / sizes


def prepare(case, seed):
    kind = case["kind"]
    if kind == "rows":  # the state and the relative states as the reference's driver holds them, six values a particle
        s, eps, _ = _system(case["workload"], case["n"], seed)
        return {"case": case, "eps": eps, "state": np.ascontiguousarray(s.T), "out": np.zeros(6 * case["n"])}
    solver = BIASolver(device=0)
    if kind == "ensemble":
        s, eps = _ensemble(case, seed)
        q = None
        ens = solver.ensemble(_sizes(case), eps)
        cfg = default_config(dt=case["dt"], method=METHODS[case["method"]])
    else:
        s, eps, q = _system(case["workload"], case["n"], seed)
        ens, cfg = None, None
        if "method" in case:
            cfg = default_config(eps_th=eps, dt=case["dt"], method=METHODS[case["method"]])
    if case.get("method") == "learned":
        solver.load_heads()
    if kind == "host":
        state = torch.tensor(s).pin_memory().numpy()
    else:
        state = torch.tensor(s, device="cuda")
        q = None if q is None else torch.tensor(q, device="cuda")
    torch.cuda.synchronize()
    return {"case": case, "solver": solver, "ens": ens, "cfg": cfg, "state": state, "q": q, "eps": eps}


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "step":
        st["solver"].step(st["state"], st["cfg"], q=st["q"], stats=False)
        return st["state"]
    if kind == "advance":  # the state that the step starts from is kept
        s = st["state"].clone()
        st["solver"].step(s, st["cfg"], q=st["q"], stats=False)
        return s
    if kind == "run":
        st["solver"].run(st["state"], st["cfg"], case["steps"], q=st["q"], stats=False)
        return st["state"]
    if kind == "host":
        st["solver"].run_host(st["state"], st["cfg"], 1, q=st["q"])
        return st["state"]
    if kind == "ensemble":
        st["ens"].run(st["state"], st["cfg"], case["steps"], stats=False)
        return st["state"]
    if kind == "dim":  # the check starts from the state that the BIA run has, which stays as it is
        s = st["state"].clone()
        st["solver"].dim_integrate(s, 0.5 * st["eps"], 0.0, case["t"])
        return s
    if kind == "rows":
        n, s = case["n"], st["state"]
        acc = np.zeros((6, n))
        for i in range(n):
            find_dxyuv_kernel(METHODS[case["method"]], n, i + 1, st["eps"], case["dt"], 18, *acc, (s[i] - s).reshape(-1), st["out"])
        acc[:3] += s[:, 3:].T * case["dt"]
        st["state"] = s + acc.T
        return st["state"]
    return st["solver"].invariance(st["state"], st["eps"], q=st["q"])


# ---- what a pass cannot do without -------------------------------------------------------

# FP64 operations of one pair (+ - * / sqrt = 1, FMA = 2): differences, 1/r, energy, a solve of the
# orbit by its series and the composition and two sums of the six displacements; a direct sum's
# and an inverse distance's
PAIR_FLOPS, RKF_FLOPS, FORCE_FLOPS, DISTANCE_FLOPS = 142, 4000, 20, 11


def work(case):
    kind = case["kind"]
    steps = case.get("steps", 1)
    if kind == "ensemble":
        sizes = _sizes(case).astype(np.float64)
        n, pairs = float(sizes.sum()), float((sizes * (sizes - 1) / 2).sum())
    else:
        n, pairs = float(case["n"]), case["n"] * (case["n"] - 1) / 2.0
    per = RKF_FLOPS if case.get("method") == "rkf" else PAIR_FLOPS
    if kind == "rows":  # each call's relative states in, its displacements out
        return {"bytes": 96.0 * n * n, "flops": pairs * per}
    if kind == "invariants":
        return {"bytes": 56.0 * n, "flops": DISTANCE_FLOPS * pairs}
    if kind == "dim":  # six derivatives of each accepted step; about one step in 1e-4 of these systems' time
        return {"bytes": 96.0 * n, "flops": max(4.0, case["t"] / 1e-4) * 6 * n * (n - 1) * FORCE_FLOPS}
    return {"bytes": 96.0 * n * steps, "flops": pairs * per * steps}


# ---- the same in plain torch -------------------------------------------------------------


def _stumpff(x):
    small = x.abs() <= 0.3
    y = torch.where(small, x, 0.0)
    c2 = torch.full_like(y, 1.0 / math.factorial(22))
    c3 = torch.full_like(y, 1.0 / math.factorial(23))
    for k in range(9, -1, -1):
        c2 = 1.0 / math.factorial(2 * k + 2) - y * c2
        c3 = 1.0 / math.factorial(2 * k + 3) - y * c3
    z = torch.where(small, 1.0, x)
    a = z.abs().sqrt()
    pos = z > 0
    b = torch.where(pos, 1.0, a).clamp(max=600.0)
    k2 = torch.where(pos, 2.0 * torch.sin(0.5 * a) ** 2, 2.0 * torch.sinh(0.5 * b) ** 2) / z.abs()
    k3 = torch.where(pos, a - torch.sin(a), torch.sinh(b) - b) / (z.abs() * a)
    c2, c3 = torch.where(small, c2, k2), torch.where(small, c3, k3)
    return 1.0 - x * c2, 1.0 - x * c3, c2, c3


def _orbit(eps, dt, r2, rg, g2):
    """f - 1, g - dt, f', g' - 1 of r'' = eps r / |r|^3 over dt (universal variables, Laguerre's iteration)."""
    mu = -eps
    r0 = r2.sqrt()
    beta = 2.0 * mu / r0 - g2
    # a start that is not far above the root, where the hyperbolic functions would swamp the iteration
    s = dt / (r0 + torch.where(beta < 0, (-beta).clamp(min=0.0).sqrt() * dt, 0.0))
    for _ in range(16):
        c0, c1, c2, c3 = _stumpff(beta * s * s)
        f = r0 * s * c1 + rg * s * s * c2 + mu * s ** 3 * c3 - dt
        f1 = r0 * c0 + rg * s * c1 + mu * s * s * c2
        f2 = rg * c0 + (mu - beta * r0) * s * c1
        s = s - 5.0 * f / (f1 + (16.0 * f1 * f1 - 20.0 * f * f2).abs().sqrt())
    c0, c1, c2, c3 = _stumpff(beta * s * s)
    rt = r0 * c0 + rg * s * c1 + mu * s * s * c2
    return -mu * s * s * c2 / r0, -mu * s ** 3 * c3, -mu * s * c1 / (rt * r0), -mu * s * s * c2 / rt


def _displacements(a, b, eps, dt, skip):
    """Half the displacement from free motion of particles a (6, p) against each of b (6, m): (6, p, m).
    skip: the pairs that are left out."""
    r = [a[k][:, None] - b[k][None, :] for k in range(6)]
    r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2]
    r2[skip] = 1.0
    rg = r[0] * r[3] + r[1] * r[4] + r[2] * r[5]
    g2 = r[3] * r[3] + r[4] * r[4] + r[5] * r[5]
    # f and g by their Taylor series in dt where the step is short against the pair's times
    i2 = 1.0 / r2
    mu = -eps
    u = mu * i2 * i2.sqrt()
    p = rg * i2
    q = g2 * i2 - u
    hard = (u.abs() + p * p + g2 * i2) * (dt * dt) > 2.5e-7
    w = 3.0 * q - 15.0 * p * p + u
    fm1 = u * (dt * dt) * (-0.5 + dt * (0.5 * p + dt * (w / 24.0 + dt * p * (7.0 * p * p - 3.0 * q - u) / 8.0)))
    gmt = u * dt ** 3 * (-1.0 / 6.0 + dt * (0.25 * p + dt * (9.0 * q - 45.0 * p * p + u) / 120.0))
    fd = u * dt * (-1.0 + dt * (1.5 * p + dt * (w / 6.0 + dt * p * (7.0 * p * p - 3.0 * q - u) * 0.625)))
    gd1 = u * (dt * dt) * (-0.5 + dt * (p + dt * (9.0 * q - 45.0 * p * p + u) / 24.0))
    at = torch.nonzero(hard.reshape(-1)).squeeze(1)
    if at.numel():
        e = eps.expand_as(r2).reshape(-1)[at] if isinstance(eps, torch.Tensor) else torch.full_like(r2.reshape(-1)[at], eps)
        parts = _orbit(e, dt, r2.reshape(-1)[at], rg.reshape(-1)[at], g2.reshape(-1)[at])
        for whole, part in zip((fm1, gmt, fd, gd1), parts):
            whole.view(-1)[at] = part
    for c in (fm1, gmt, fd, gd1):
        c[skip] = 0.0
    return [0.5 * (fm1 * r[k] + gmt * r[3 + k]) for k in range(3)] + [0.5 * (fd * r[k] + gd1 * r[3 + k]) for k in range(3)]


def _step(s, eps, dt, q=None):
    n = s.shape[1]
    out = torch.zeros_like(s)
    rows = max(1, min(n, (1 << 25) // n))
    ids = torch.arange(n, device=s.device)
    for i in range(0, n, rows):
        a = s[:, i : i + rows]
        e = eps if q is None else eps * q[i : i + rows, None] * q[None, :]
        h = _displacements(a, s, e, dt, ids[i : i + rows, None] == ids[None, :])
        for k in range(6):
            out[k, i : i + rows] = h[k].sum(1)
    out[:3] += s[3:] * dt
    return s + out


def _force(s, eps):
    n = s.shape[1]
    d = [s[k][:, None] - s[k][None, :] for k in range(3)]
    r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
    r2.fill_diagonal_(1.0)
    w = eps / (r2 * r2.sqrt())
    return torch.stack([s[3], s[4], s[5]] + [(w * d[k]).sum(1) for k in range(3)])


def _integrate(s, eps, t):
    """Gragg's modified midpoint rule over equal steps, extrapolated."""
    steps = max(1, int(math.ceil(t / 2.5e-4)))
    h = t / steps
    seq = (2, 4, 6, 8, 10, 12, 14)
    for _ in range(steps):
        f0 = _force(s, eps)
        table = []
        for j, m in enumerate(seq):
            d = h / m
            # z - s, so that the sums keep the digits of the small increments
            z0, z1 = torch.zeros_like(s), d * f0
            for _k in range(1, m):
                z0, z1 = z1, z0 + 2.0 * d * _force(s + z1, eps)
            new = [0.5 * (z0 + z1 + d * _force(s + z1, eps))]
            for k in range(j):
                x = (seq[j] / seq[j - k - 1]) ** 2
                new.append(new[k] + (new[k] - table[k]) / (x - 1.0))
            table = new
        s = s + table[-1]
    return s


def _invariants(s, eps, q):
    n = s.shape[1]
    x, y, z, u, v, w = s
    pe = torch.zeros((), dtype=torch.float64, device=s.device)
    ids = torch.arange(n, device=s.device)
    rows = max(1, (1 << 26) // n)
    for i in range(0, n, rows):
        r2 = sum((s[k, i : i + rows, None] - s[k][None, :]) ** 2 for k in range(3))
        w1 = torch.where(ids[i : i + rows, None] < ids[None, :], 1.0 / r2.sqrt(), 0.0)
        pe += (w1 if q is None else w1 * q[i : i + rows, None] * q[None, :]).sum()
    out = {"KE": (u * u + v * v + w * w).sum(), "PE": eps * pe, "Lx": (y * w - z * v).sum(), "Ly": (z * u - x * w).sum(),
           "Lz": (x * v - y * u).sum(), "Ua": u.sum(), "Va": v.sum(), "Wa": w.sum(), "Xa": x.sum(), "Ya": y.sum(), "Za": z.sum()}
    out = {k: float(a) for k, a in out.items()}
    for k, a in (("Lx", (y, w, z, v)), ("Ly", (z, u, x, w)), ("Lz", (x, v, y, u)), ("Ua", (u,)), ("Va", (v,)), ("Wa", (w,)),
                 ("Xa", (x,)), ("Ya", (y,)), ("Za", (z,))):
        # sums that cancel to rounding have no digits to compare
        size = float((a[0].abs() * a[1].abs() + a[2].abs() * a[3].abs()).sum() if len(a) == 4 else a[0].abs().sum())
        if abs(out[k]) < 1e-9 * size:
            out[k] = None
    return out


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "ensemble":
        s, eps = _ensemble(case, seed)
        s, at, parts = torch.tensor(s, device=dev), 0, []
        for n, e in zip(_sizes(case), eps):
            a = s[:, at : at + int(n)]
            for _ in range(case["steps"]):
                a = _step(a, float(e), case["dt"])
            parts.append(a)
            at += int(n)
        return torch.cat(parts, 1)
    s, eps, q = _system(case["workload"], case["n"], seed)
    s = torch.tensor(s, device=dev)
    q = None if q is None else torch.tensor(q, device=dev)
    if kind == "dim":
        if case["t"] * case["n"] > 20.0:
            return None
        return _integrate(s, 0.5 * eps, case["t"])
    if kind == "invariants":
        return _invariants(s, eps, q)
    for _ in range(case.get("steps", 1)):
        s = _step(s, eps, case["dt"], q)
    if kind == "rows":
        return s.T.cpu().numpy()
    return s.cpu().numpy() if kind == "host" else s
