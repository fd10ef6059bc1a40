"""Workloads of the force library, timed through its public entry points.

Each case is a dict of plain values; `kind` names the call a program makes:

  gravity   Engine.gravity on CUDA tensors: octree build + Barnes-Hut walk of every particle
            (host: the same on NumPy arrays, the reference's own calling convention)
  substeps  Engine.gravity on CUDA tensors over one long step: a build with everybody active,
            then sub-steps that drift the particles and refit the tree for the fast ones
  direct    Engine.gravity_direct on CUDA tensors: the exact float64 sum
  forces    gf_accelerations_dev, two full evaluations of a particle set (the initial one, and
            the next one after a drift): gravity + neighbour search + smoothing lengths + SPH,
            in the plain form (the reference's arithmetic) or the mixed one (float32 SPH,
            quadrupoles under the relative opening criterion)
  sph       galaxy_formation_gb300.sph on NumPy arrays: NeighbourFinder.find (a fresh search, and
            a reselection after a drift) and sph_forces
  steps     gf_sim_init, gf_sim_step, gf_sim_read: the hierarchical step loop, plain form
  blocks    gf_sim_init, gf_sim_blocks, gf_sim_read: the block time steps, mixed form

Particle sets (drawn on the GPU from the seed): `cloud` is the rotating 1/r sphere the
simulations start from, `disk` the collapsed exponential disk in a 1/r halo, with `clumps`
Plummer spheres carved out of the disk gas.
"""

import ctypes
import math

import numpy as np
import torch

from galaxy_formation_gb300 import _lib, params, sph
from galaxy_formation_gb300.engine import Engine

M_TOT = 2.8e11 / params.MSUN
F_BARYON = 0.16
R0 = 100.0 / params.KPC
RD, Z0, A_CLUMP = 3.0 / params.KPC, 0.3 / params.KPC, 0.2 / params.KPC
DRIFT = 2e-4          # time between two evaluations of a set (code units): a small step
BLOCK_LEVELS = 6      # block time steps over 2^5 finest sub-steps


def listed():
    return [
        # the reference's default simulation (5,000 gas + 5,000 dark matter): smallest calls,
        # a chain of short launches
        {"name": "gravity_cloud_10k", "kind": "gravity", "set": "cloud", "n_gas": 5000, "n_dm": 5000, "host": False},
        # the same call as the reference's own Python makes it: NumPy arrays in and out
        {"name": "gravity_host_50k", "kind": "gravity", "set": "cloud", "n_gas": 24999, "n_dm": 25002, "host": True},
        # a large simulation's gravity: the 4M rotating cloud
        {"name": "gravity_cloud_4M", "kind": "gravity", "set": "cloud", "n_gas": 2000000, "n_dm": 2000000,
         "host": False},
        # one long step of a caller that drives the time stepping itself: few active particles
        # on a refitted tree
        {"name": "substeps_disk_200k", "kind": "substeps", "set": "disk", "n_gas": 100000, "n_dm": 100000, "steps": 8,
         "active": 0.06},
        # accuracy checks and small systems: the exact sum, odd size
        {"name": "direct_20k", "kind": "direct", "set": "cloud", "n_gas": 10007, "n_dm": 9994},
        # the default simulation's full force evaluation
        {"name": "forces_cloud_10k", "kind": "forces", "set": "cloud", "n_gas": 5000, "n_dm": 5000, "mixed": False},
        # the benchmark snapshot in the reference's arithmetic
        {"name": "forces_disk_1M", "kind": "forces", "set": "disk", "n_gas": 500000, "n_dm": 500000, "mixed": False},
        # the benchmark snapshot in the mixed form, as the benchmark's headline runs it
        {"name": "forces_mixed_disk_1M", "kind": "forces", "set": "disk", "n_gas": 500000, "n_dm": 500000,
         "mixed": True},
        # gas only, clumped over six decades of density (ragged neighbourhoods), plain form
        {"name": "forces_clumps_150k", "kind": "forces", "set": "disk", "n_gas": 150001, "n_dm": 0, "clumps": 200,
         "mixed": False},
        # the SPH module alone, as the reference's simulation.py calls it with NumPy arrays
        {"name": "sph_host_60k", "kind": "sph", "set": "disk", "n_gas": 60011, "n_dm": 0},
        # a short simulation: initial forces and one hierarchical long step
        {"name": "steps_disk_200k", "kind": "steps", "set": "disk", "n_gas": 100000, "n_dm": 100000, "steps": 1},
        # the same with block time steps in the mixed form: two blocks replayed as CUDA graphs
        {"name": "blocks_disk_200k", "kind": "blocks", "set": "disk", "n_gas": 100000, "n_dm": 100000, "blocks": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gravity", "gravity", "substeps", "direct", "forces", "forces", "forces", "sph", "steps",
                       "blocks"])
    # particles of a drawn case, over the range of the listed ones of its kind
    lo, hi = {"gravity": (3000, 2000000), "substeps": (5000, 500000), "direct": (500, 40000),
              "forces": (3000, 1000000), "sph": (1000, 200000), "steps": (4000, 200000),
              "blocks": (4000, 200000)}[kind]
    n = _log_int(rng, lo, hi)
    c = {"kind": kind, "set": rng.choice(["cloud", "disk"])}
    gas = 1.0 if kind == "sph" else rng.choice([0.5, 0.5, rng.uniform(0.2, 0.9), 1.0])
    c["n_gas"] = max(200, int(n * gas))
    c["n_dm"] = 0 if gas == 1.0 else max(1, n - c["n_gas"])
    if c["set"] == "disk" and n > 20000 and rng.random() < 0.3:
        c["clumps"] = rng.randint(3, 200)
    if kind == "gravity":
        c["host"] = n < 300000 and rng.random() < 0.3
        c["theta"] = rng.choice([0.7, 0.7, 0.5, 0.9])
    elif kind == "substeps":
        c["steps"] = rng.randint(2, 8)
        c["active"] = round(math.exp(rng.uniform(math.log(0.002), math.log(0.9))), 4)
    elif kind == "forces":
        c["mixed"] = rng.random() < 0.4
    elif kind == "steps":
        c["steps"] = 1
    elif kind == "blocks":
        c["blocks"] = rng.randint(1, 2)
    return c


# ------------------------------------------------------------------------ particle sets


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _ball(n, g):
    v = _randn(g, n, 3)
    v = v / v.norm(dim=1, keepdim=True)
    return v * R0 * _rand(g, n, 1).sqrt()


def _sech2(n, g):
    return Z0 * torch.atanh((2 * _rand(g, n) - 1).clamp(-1 + 1e-12, 1 - 1e-12))


def _disk_radii(n, rmax, g):
    r = -RD * torch.log(_rand(g, n).clamp_min(1e-300) * _rand(g, n).clamp_min(1e-300))
    return torch.remainder(r, rmax)


def _disk_points(n, rmax, g):
    r, ph = _disk_radii(n, rmax, g), 2 * math.pi * _rand(g, n)
    return torch.stack([r * torch.cos(ph), r * torch.sin(ph), _sech2(n, g)], 1)


def particles(case, seed):
    """pos, vel (n,3), mass, kind (int8: 0 gas, 2 dark matter; gas first), u of a case, on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)
    ng, nd = case["n_gas"], case["n_dm"]
    n = ng + nd
    mass = torch.empty(n, dtype=torch.float64, device="cuda")
    mass[:ng] = F_BARYON * M_TOT / ng
    if nd:
        mass[ng:] = (1 - F_BARYON) * M_TOT / nd
    else:
        mass[:] = M_TOT / ng
    kind = torch.zeros(n, dtype=torch.int8, device="cuda")
    kind[ng:] = params.DM
    u = torch.zeros(n, dtype=torch.float64, device="cuda")
    if case["set"] == "cloud":
        pos = torch.cat([_ball(ng, g), _ball(nd, g)])
        rotating = 0
        u[:ng] = 1e4 * params.U_PER_K
    else:
        n_disk = int(round(0.6 * ng))
        clumps = int(case.get("clumps", 0))
        each = max(1, ng // 1000) if clumps else 0
        clumps = min(clumps, n_disk // max(1, each))
        parts = [_disk_points(n_disk - clumps * each, 12 * RD, g)]
        if clumps:  # Plummer spheres: r = a / sqrt(U^(-2/3) - 1)
            cen = _disk_points(clumps, 6 * RD, g)
            rr = A_CLUMP / ((1e-6 + 0.998 * _rand(g, clumps, each)).pow(-2.0 / 3.0) - 1.0).sqrt()
            d = _randn(g, clumps, each, 3)
            d = d / d.norm(dim=2, keepdim=True)
            parts.append((cen[:, None, :] + d * rr[..., None]).reshape(-1, 3))
        parts += [_ball(ng - n_disk, g), _ball(nd, g)]
        pos = torch.cat(parts)
        rotating = n_disk
        u[:ng] = torch.exp(math.log(1e4) + math.log(100.0) * _rand(g, ng)) * params.U_PER_K
    r = pos.norm(dim=1)
    order = torch.argsort(r)
    inside = torch.cumsum(order < ng, 0)  # gas particles within each radius (integers: exact sums)
    menc = torch.empty_like(r)
    menc[order] = mass[0] * inside + mass[-1] * (torch.arange(1, n + 1, device="cuda") - inside)
    vc = (menc / r.clamp_min(1e-6)).sqrt()
    rcyl = torch.hypot(pos[:, 0], pos[:, 1]).clamp_min(1e-30)
    phi_hat = torch.stack([-pos[:, 1] / rcyl, pos[:, 0] / rcyl, torch.zeros_like(r)], 1)
    rot = 0.05 / 0.47 * rcyl / r.clamp_min(1e-6)
    rot[:rotating] = 1.0
    vel = (rot * vc)[:, None] * phi_hat + 0.1 * vc[:, None] * _randn(g, n, 3) / math.sqrt(3.0)
    vel = vel - (mass[:, None] * vel).sum(0) / mass.sum()
    return {"pos": pos.contiguous(), "vel": vel.contiguous(), "mass": mass, "kind": kind, "u": u}


def _active_masks(case, seed, pos):
    """The fast particles of a sub-step: mostly the inner ones, where the steps are short."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 99)
    n = len(pos)
    score = torch.log(pos.norm(dim=1).clamp_min(1e-12)) + 0.5 * _randn(g, n)
    fast = torch.zeros(n, dtype=torch.uint8, device="cuda")
    fast[torch.argsort(score)[:max(1, int(case["active"] * n))]] = 1
    return fast


# ------------------------------------------------------------------------------ the calls


def _options(lib, mixed):
    """The options of the plain form, or of the benchmark's mixed form."""
    for key, value in [(_lib.OPT_SPH_FLOAT32, 1 if mixed else 0), (_lib.OPT_GRAVITY_QUAD, 1 if mixed else 0),
                       (_lib.OPT_HGUESS, 0), (_lib.OPT_WALK_MERGE, 40 if mixed else 0),
                       (_lib.OPT_GRAVITY_REL_MONO, 1.5e-4 if mixed else 0.0),
                       (_lib.OPT_GRAVITY_REL, 4e-3 if mixed else 0.0)]:
        _lib.check(lib.gf_set_option(key, value))


def _mixed(case):
    return case["kind"] == "blocks" or bool(case.get("mixed"))


def prepare(case, seed):
    kind = case["kind"]
    d = particles(case, seed)
    n = len(d["mass"])
    st = {"case": dict(case), "engine": Engine()}
    st["lib"] = st["engine"].lib
    _options(st["lib"], _mixed(case))
    if kind in ("steps", "blocks", "sph") or case.get("host"):
        st["d"] = {k: v.cpu().numpy() for k, v in d.items()}
    else:
        st["d"] = d
        st["acc"] = torch.zeros_like(d["pos"])
    if kind == "substeps":
        st["active"] = _active_masks(case, seed, d["pos"])
    if kind == "forces":
        st["acc2"] = torch.zeros_like(d["pos"])
        st["dt"] = torch.zeros_like(d["mass"])
        st["dt2"] = torch.zeros_like(d["mass"])
    torch.cuda.synchronize()
    return st


def _run_forces(st):
    lib, d, mixed = st["lib"], st["d"], _mixed(st["case"])
    theta = 0.55 if mixed else params.THETA
    n = len(d["mass"])
    stream = torch.cuda.current_stream().cuda_stream or 1
    # an unrelated particle set: no previous smoothing lengths, no previous error scale
    _lib.check(lib.gf_set_option(_lib.OPT_FORGET_H, 1))
    if mixed:
        _lib.check(lib.gf_set_option(_lib.OPT_GRAVITY_REL, 4e-3))
    pos = d["pos"]
    for acc, dt in ((st["acc"], st["dt"]), (st["acc2"], st["dt2"])):
        _lib.check(lib.gf_accelerations_dev(
            n, pos.data_ptr(), d["vel"].data_ptr(), d["mass"].data_ptr(), d["kind"].data_ptr(), d["u"].data_ptr(),
            theta, params.EPS, params.GAMMA, sph.ALPHA, sph.BETA, None, 1, 1, 1, acc.data_ptr(), dt.data_ptr(),
            stream))
        pos = d["pos"] + DRIFT * d["vel"]
    return {"acc": st["acc"], "dt": st["dt"], "acc2": st["acc2"], "dt2": st["dt2"]}


def _run_sph(st):
    d = st["d"]
    n = len(d["mass"])
    gas = np.arange(n)
    find = sph.NeighbourFinder(n)
    out = {}
    pos = d["pos"]
    for name, fresh in (("fresh", True), ("again", False)):
        dist, nb = find.find(gas, pos, fresh)
        h = np.maximum(0.5 * dist[:, -1], 0.5 * params.EPS)
        rho, acc, dudt, dt = np.empty(n), np.empty((n, 3)), np.empty(n), np.empty(n)
        sph.sph_forces(pos, d["vel"], d["mass"], nb, h, d["u"], params.GAMMA, sph.ALPHA, sph.BETA, rho, acc, dudt, dt)
        out[name] = {"nb": nb, "dist": dist, "rho": rho, "acc": acc, "dudt": dudt, "dt": dt}
        pos = pos + DRIFT * d["vel"]
    return out


def _run_simulation(st):
    lib, d, case = st["lib"], st["d"], st["case"]
    n = len(d["mass"])
    theta = 0.55 if _mixed(case) else params.THETA
    _lib.check(lib.gf_sim_init(n, d["pos"], d["vel"], d["mass"], d["kind"], d["u"], theta, params.EPS, params.GAMMA,
                               sph.ALPHA, sph.BETA))
    taken, sub, upd = ctypes.c_double(), ctypes.c_int(), ctypes.c_double()
    if case["kind"] == "steps":
        for _ in range(case["steps"]):
            _lib.check(lib.gf_sim_step(1.0, ctypes.byref(taken), ctypes.byref(sub)))
    else:
        _lib.check(lib.gf_sim_blocks(case["blocks"], BLOCK_LEVELS, ctypes.byref(upd)))
    out = {"pos": np.empty((n, 3)), "vel": np.empty((n, 3)), "acc": np.empty((n, 3)), "dt": np.empty(n)}
    t = ctypes.c_double()
    _lib.check(lib.gf_sim_read(out["pos"].ctypes.data, out["vel"].ctypes.data, out["acc"].ctypes.data,
                               out["dt"].ctypes.data, ctypes.byref(t)))
    out["t"] = t.value
    return out


def run(st):
    case, kind, d, eng = st["case"], st["case"]["kind"], st["d"], st["engine"]
    theta = case.get("theta", params.THETA)
    if kind == "gravity":
        acc = np.zeros_like(d["pos"]) if case.get("host") else st["acc"]
        eng.gravity(d["pos"], d["mass"], acc, theta, params.EPS)
        return acc
    if kind == "substeps":
        acc, pos = st["acc"], d["pos"]
        eng.gravity(pos, d["mass"], acc, theta, params.EPS)
        for _ in range(case["steps"]):
            pos = pos + DRIFT * d["vel"]
            eng.gravity(pos, d["mass"], acc, theta, params.EPS, st["active"], False)
        return acc
    if kind == "direct":
        return eng.gravity_direct(d["pos"], d["mass"], params.EPS)
    if kind == "forces":
        return _run_forces(st)
    if kind == "sph":
        return _run_sph(st)
    return _run_simulation(st)


# ------------------------------------------------------- what a pass cannot do without


def _gravity_flops(n, theta, active=1.0):
    # a Barnes-Hut list of about 70 log2(n) entries per particle at opening angle 0.7 (measured:
    # 1400 at 1M), 20 flops each
    return 20.0 * 70.0 * math.log2(max(n, 2)) * (0.7 / theta) ** 2 * n * active


def _sph_flops(ng):
    # per gas particle: about 150 distances of the neighbour search (8 flops), 32 neighbours at
    # 20 (density) and 60 flops (forces)
    return ng * (150 * 8 + 32 * 80.0)


def work(case):
    kind, ng = case["kind"], case["n_gas"]
    n = ng + case["n_dm"]
    theta = case.get("theta", params.THETA)
    grav_bytes = n * (24 + 8 + 24)
    if kind == "gravity":
        return {"bytes": grav_bytes, "flops": _gravity_flops(n, theta)}
    if kind == "substeps":
        a = case["active"]
        return {"bytes": grav_bytes + case["steps"] * (n * (24 + 24 + 24 + 8 + 1) + a * n * 24),
                "flops": _gravity_flops(n, theta) * (1 + case["steps"] * a) + case["steps"] * 6.0 * n}
    if kind == "direct":
        return {"bytes": grav_bytes, "flops": 20.0 * n * n}
    force_bytes = n * (24 + 24 + 8 + 1 + 8 + 24 + 8)
    force_flops = _gravity_flops(n, theta) + _sph_flops(ng)
    if kind == "forces":
        return {"bytes": 2 * force_bytes + n * (24 + 24 + 24), "flops": 2 * force_flops}
    if kind == "sph":
        per = n * (24 + 24 + 8 + 8 + 32 * 16 + 8 + 24 + 8 + 8)
        return {"bytes": 2 * per, "flops": 2 * _sph_flops(n)}
    # the simulations: initial forces, one long step (or its blocks), every particle once more
    evals = 2 * case.get("steps", 1) if kind == "steps" else 1 + 2 * case["blocks"]
    return {"bytes": (1 + evals) * force_bytes, "flops": (1 + evals) * force_flops}


# -------------------------------------------------------------------- values in 64 bits


def _chunks(n, width):
    step = max(1, int(1.5e8 // max(1, width)))
    return [(a, min(n, a + step)) for a in range(0, n, step)]


def _direct64(pos, mass, rows=None):
    """Softened direct sum in float64 (rows: indices of the targets, default all)."""
    tgt = pos if rows is None else pos[rows]
    out = torch.empty_like(tgt)
    x, y, z = (pos[:, k].contiguous() for k in range(3))
    for a, b in _chunks(len(tgt), len(pos)):
        dx, dy, dz = (p[None, :] - tgt[a:b, k, None] for k, p in enumerate((x, y, z)))
        r2 = dx * dx
        r2.addcmul_(dy, dy).addcmul_(dz, dz).add_(params.EPS ** 2)
        f = mass[None, :] / (r2 * r2.sqrt())
        for k, dk in enumerate((dx, dy, dz)):
            out[a:b, k] = (f * dk).sum(1)
    return out


def _nearest64(pos, k):
    """The k nearest of every point (itself included), ascending: distances and indices."""
    n = len(pos)
    dist = torch.empty(n, k, dtype=torch.float64, device=pos.device)
    nb = torch.empty(n, k, dtype=torch.int64, device=pos.device)
    x, y, z = (pos[:, c].contiguous() for c in range(3))
    for a, b in _chunks(n, n):
        d2 = (pos[a:b, 0, None] - x[None, :]).square_()
        d2 += (pos[a:b, 1, None] - y[None, :]).square_()
        d2 += (pos[a:b, 2, None] - z[None, :]).square_()
        v, i = torch.topk(d2, k, dim=1, largest=False)
        dist[a:b], nb[a:b] = v.sqrt(), i
    return dist, nb


def _w_m4(q):
    t = (2 - q).clamp_min(0)
    return torch.where(q < 1, 1 - 1.5 * q * q + 0.75 * q ** 3, 0.25 * t ** 3)


def _dw_m4(q):
    t = (2 - q).clamp_min(0)
    return torch.where(q < 1, -3 * q + 2.25 * q * q, -0.75 * t * t)


def _sph64(pos, vel, mass, nb, h, u, gamma=5.0 / 3.0, alpha=1.0, beta=2.0):
    """Density, acceleration, du/dt and Courant step (cubic spline, Monaghan-Gingold viscosity)."""
    d = pos[:, None, :] - pos[nb]
    r2 = (d * d).sum(2)
    r = r2.sqrt()
    hi, hj = h[:, None], h[nb]
    rho = (mass[nb] * _w_m4(r / hi)).sum(1) / (math.pi * h ** 3)
    cs = (gamma * (gamma - 1) * u).sqrt()
    pr2 = (gamma - 1) * u / rho
    other = nb != torch.arange(len(pos), device=pos.device)[:, None]
    inv_r = 1 / r.clamp_min(1e-30)
    gi = _dw_m4(r / hi) * inv_r / (math.pi * hi ** 4)
    gj = _dw_m4(r / hj) * inv_r / (math.pi * hj ** 4)
    vr = ((vel[:, None, :] - vel[nb]) * d).sum(2)
    hb = 0.5 * (hi + hj)
    mu = torch.where((vr < 0) & other, hb * vr / (r2 + 0.01 * hb * hb), torch.zeros_like(r))
    visc = (-alpha * 0.5 * (cs[:, None] + cs[nb]) * mu + beta * mu * mu) / (0.5 * (rho[:, None] + rho[nb]))
    gb = 0.5 * (gi + gj)
    m = torch.where(other, mass[nb], torch.zeros_like(r))
    acc = -((m * (pr2[:, None] * gi + pr2[nb] * gj + visc * gb))[..., None] * d).sum(1)
    dudt = (m * (pr2[:, None] * gi + 0.5 * visc * gb) * vr).sum(1)
    mu_max = (-mu).amax(1).clamp_min(0)
    dt = 0.3 * h / (cs + 1.2 * (alpha * cs + beta * mu_max) + 1e-30)
    return rho, acc, dudt, dt


def _forces64(d, pos):
    acc = _direct64(pos, d["mass"])
    dt = torch.full_like(d["mass"], math.inf)
    g = torch.nonzero(d["kind"] == 0).flatten()
    if len(g) > 40:
        p, v, m, u = pos[g].contiguous(), d["vel"][g], d["mass"][g], d["u"][g]
        dist, nb = _nearest64(p, 32)
        h = (0.5 * dist[:, -1]).clamp_min(0.5 * params.EPS)
        _, a, _, dti = _sph64(p, v, m, nb, h, u)
        acc[g] += a
        dt[g] = dti
    mag = acc.norm(dim=1).clamp_min(1e-30)
    return acc, torch.minimum(0.3 * (params.EPS / mag).sqrt(), dt)


def exact(case, seed):
    """What run() returns, in plain float64 (direct sums, brute-force neighbours); None where
    the O(n^2) work would take too long, and for the simulations, whose every sub-step would
    need it."""
    kind = case["kind"]
    n = case["n_gas"] + case["n_dm"]
    if kind in ("steps", "blocks"):
        return None
    if n > (160000 if kind in ("forces", "sph") else 210000):
        return None
    d = particles(case, seed)
    if kind in ("gravity", "direct"):
        return _direct64(d["pos"], d["mass"])
    if kind == "substeps":
        pos = d["pos"]
        acc = _direct64(pos, d["mass"])
        for _ in range(case["steps"]):
            pos = pos + DRIFT * d["vel"]
        rows = torch.nonzero(_active_masks(case, seed, d["pos"])).flatten()
        acc[rows] = _direct64(pos, d["mass"], rows)
        return acc
    if kind == "forces":
        acc, dt = _forces64(d, d["pos"])
        acc2, dt2 = _forces64(d, d["pos"] + DRIFT * d["vel"])
        return {"acc": acc, "dt": dt, "acc2": acc2, "dt2": dt2}
    out = {}
    # the search runs on the same float64 positions the host call gets
    pos = d["pos"]
    for name in ("fresh", "again"):
        dist, nb = _nearest64(pos, 32)
        h = (0.5 * dist[:, -1]).clamp_min(0.5 * params.EPS)
        rho, acc, dudt, dt = _sph64(pos, d["vel"], d["mass"], nb, h, d["u"])
        out[name] = {"nb": None, "dist": dist, "rho": rho, "acc": acc, "dudt": dudt, "dt": dt}
        pos = pos + DRIFT * d["vel"]
    return out
