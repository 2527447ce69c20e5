"""The solves that the performance of this framework is measured on.

Every case goes through the public Python entry points (Context, Server, workloads) on synthetic
inputs of the shapes and distributions that the benchmark configurations and the tests use. The
grids and counters of a solve are whole numbers (fixed-point deposits), so they are the same on
every run of the same inputs.

Kinds of case:
  solve      one Context.solve of a config-model body on one of the three paths
  reference  the ballistic runner's work on the reference model: solve with per-particle rows,
             then the velocity record that the collisional phase reads
  advanced   the collisional runner's work on the reference model: fits from the recorded speeds,
             then the solve with collisions
  two_phase  the config-model collisional pipeline: phase 1 with speed histograms, degree-6 fits,
             phase 2 with collisions
  batch      independent exospheres of uneven size through one Server
  thermal    the thermal column model that makes the temperature map
  shadow     the Monte Carlo shadow flux of a cratered body
"""
from __future__ import annotations

import math

import numpy as np

import dsmc_suite_b200 as D
from dsmc_suite_b200 import _native as N
from dsmc_suite_b200 import workloads as W

PATHS = {"fast_fp32": N.PATH_FAST_FP32, "fast_fp64": N.PATH_FAST_FP64, "plain_fp64": N.PATH_PLAIN_FP64}

# Mean steps of a particle's life per body at dt 2 s (lives end by night-side landing, escape or
# the 20,000-step cap), for the operation counts of work() only.
LIFE_STEPS = {"ceres": 7000, "europa": 2400, "moon": 2300, "reference": 13000, "advanced": 70000}
FLOPS_PER_STEP = 60   # the reference's Verlet update, cell index, photolysis and deposit


def listed():
    return [
        # a smoke-sized solve, as an interactive user or a test suite runs: latency alone
        {"name": "ceres_512", "kind": "solve", "path": "fast_fp32", "body": "ceres", "n": 512,
         "hd": 50, "rows": False},
        # the smallest benchmark configuration, with the per-particle rows that the .dat files hold
        {"name": "ceres_10k_rows", "kind": "solve", "path": "fast_fp32", "body": "ceres",
         "n": 10_000, "hd": 50, "rows": True},
        # the median request of the batched and served workloads, on a short-hop body
        {"name": "moon_300k", "kind": "solve", "path": "fast_fp32", "body": "moon", "n": 300_007,
         "hd": 37, "rows": False},
        # a production solve: every slot of the GPU busy for many particle lives
        {"name": "ceres_20m", "kind": "solve", "path": "fast_fp32", "body": "ceres",
         "n": 20_000_000, "hd": 50, "rows": False},
        # the FP64 engine that FP32 results are checked against at size
        {"name": "europa_1m_fp64", "kind": "solve", "path": "fast_fp64", "body": "europa",
         "n": 1_000_000, "hd": 50, "rows": False},
        # the reference-order FP64 path, the default of the drop-in runners
        {"name": "ceres_100k_plain", "kind": "solve", "path": "plain_fp64", "body": "ceres",
         "n": 100_000, "hd": 50, "rows": False},
        # `dsmc`: the reference's own physics, phase 1
        {"name": "reference_5k", "kind": "reference", "path": "fast_fp32", "n": 5_000},
        # `dsmc-adv`: the reference's own physics, phase 2
        {"name": "advanced_500", "kind": "advanced", "path": "fast_fp32", "n": 500},
        # the collisional pipeline of the benchmark configurations
        {"name": "two_phase_1m", "kind": "two_phase", "n1": 1_000_000, "n2": 1_000_000},
        # a batch of uneven exospheres in one work queue
        {"name": "batch_16", "kind": "batch", "count": 16, "mix": 20261203},
        # the temperature map of the standard grid
        {"name": "thermal_36x72", "kind": "thermal", "ftd": 36, "ffd": 72, "n_substep": 5},
        # the shadow flux of a cratered mesh over one rotation
        {"name": "shadow_20k", "kind": "shadow", "nlevel": 5, "tt": 24, "nmonte": 50},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve"] * 5 + ["reference", "advanced", "two_phase", "batch", "thermal", "shadow"])
    if kind == "solve":
        path = rng.choice(["fast_fp32"] * 4 + ["fast_fp64", "plain_fp64"])
        most = {"fast_fp32": 15_000_000, "fast_fp64": 6_000_000, "plain_fp64": 500_000}[path]
        n = _log_int(rng, 256, most)
        return {"kind": kind, "path": path, "body": rng.choice(["ceres", "europa", "moon"]), "n": n,
                "hd": rng.randint(20, 60), "rows": n < 200_000 and rng.random() < 0.3}
    if kind == "reference":
        return {"kind": kind, "path": rng.choice(["fast_fp32", "fast_fp32", "fast_fp64"]),
                "n": _log_int(rng, 500, 10_000)}
    if kind == "advanced":
        return {"kind": kind, "path": rng.choice(["fast_fp32", "fast_fp32", "fast_fp64"]),
                "n": _log_int(rng, 100, 1000)}
    if kind == "two_phase":
        return {"kind": kind, "n1": _log_int(rng, 50_000, 1_500_000), "n2": _log_int(rng, 20_000, 3_000_000)}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(2, 24), "mix": rng.randrange(1, 2**31)}
    if kind == "thermal":
        return {"kind": kind, "ftd": rng.randint(12, 72), "ffd": rng.randint(24, 120),
                "n_substep": rng.randint(2, 8)}
    return {"kind": kind, "nlevel": rng.randint(3, 5), "tt": rng.randint(4, 24), "nmonte": rng.randint(8, 50)}


# ------------------------------------------------------------------------------------------


def _config(case, rng):
    """A config-model body: T_ss and sub-solar longitude near the published ones, its own seed."""
    R, GM = W.BODIES[case["body"]]
    p = N.params_config(N.RUNNER_BALLISTIC, R, GM, case["hd"], int(rng.integers(1, 2**63)))
    sun = W.sun_vector(float(rng.uniform(0.0, 2.0 * math.pi)))
    p.sun[0], p.sun[1], p.sun[2] = sun
    return p, W.config_surface(sun, float(rng.uniform(215.0, 255.0)))


def _reference_problem(rng, runner):
    """The reference's parameters on a map with a cold night side and cold poles (freeze scans)."""
    p = N.params_reference(runner, 36, 72)
    p.seed = int(rng.integers(1, 2**63))
    T = N.latlon_temperature(36, 72, T_ss=float(rng.uniform(225.0, 245.0)), T_floor=60.0)
    T[:2, :] = 50.0
    T[-2:, :] = 50.0
    return p, N.SurfaceInputs(T_map=T)


def _speeds_per_cell(record, p, most=50):
    """At most `most` recorded speeds per cell in [td][fd][ht] order, as the collisional runner
    groups the velocity record of phase 1."""
    v, td, fd, ht = record
    keep = (td < p.ftd) & (fd < p.ffd) & (ht < p.hd)
    cell = (td[keep].astype(np.int64) * p.ffd + fd[keep]) * p.hd + ht[keep]
    speed = np.sqrt((v[keep] ** 2).sum(1))
    order = np.argsort(cell, kind="stable")
    cell, speed = cell[order], speed[order]
    first = np.searchsorted(cell, cell)
    rank = np.arange(cell.size) - first
    fits = rank < most
    speeds = np.zeros((p.ncell, most))
    counts = np.zeros(p.ncell, dtype=np.int32)
    speeds[cell[fits], rank[fits]] = speed[fits]
    np.add.at(counts, cell[fits], 1)
    return speeds, counts


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "solve":
        p, surf = _config(case, rng)
        return {"case": case, "ctx": D.Context(0), "params": p, "surface": surf}
    if kind == "reference":
        p, surf = _reference_problem(rng, N.RUNNER_BALLISTIC)
        return {"case": case, "ctx": D.Context(0), "params": p, "surface": surf}
    if kind == "advanced":
        # phase 1 is behind such a program: its density and velocity record are read from files
        ctx = D.Context(0)
        p1, surf = _reference_problem(rng, N.RUNNER_BALLISTIC)
        den = ctx.solve(N.PATH_FAST_FP32, p1, surf, 1000)["density"]
        p = N.params_reference(N.RUNNER_ADVANCED, 36, 72)
        p.seed = p1.seed
        speeds, counts = _speeds_per_cell(ctx.velocity_record(300), p)
        n_bg = den.astype(np.float64).ravel() / N.FIXED_SCALE * 1e10
        return {"case": case, "ctx": ctx, "params": p, "surface": surf, "n_bg": n_bg,
                "speeds": speeds, "counts": counts}
    if kind == "two_phase":
        return {"case": case, "ctx": D.Context(0), "seed": int(rng.integers(1, 2**63)),
                "sun": W.sun_vector(float(rng.uniform(0.0, 2.0 * math.pi))),
                "T_ss": float(rng.uniform(225.0, 245.0))}
    if kind == "batch":
        srv = D.Server(0, hbm_budget=4 * 10**9, max_requests=4096)
        # bodies, sizes, shells and maps by the case's mix; the particles' streams by the seed
        mix = np.random.default_rng(case["mix"])
        problems = [W.random_instance(mix, k) for k in range(case["count"])]
        for q in problems:
            q.params.seed = int(rng.integers(1, 2**63))
        return {"case": case, "server": srv, "problems": problems}
    if kind == "thermal":
        tp = N.ThermalParams.default()
        tp.n_substep = case["n_substep"]
        lat = (np.arange(case["ftd"]) + 0.5) / case["ftd"] * math.pi - math.pi / 2
        lon = (np.arange(case["ffd"]) + 0.5) / case["ffd"] * 2 * math.pi
        flux = 200.0 * np.cos(lat)[:, None] * np.clip(np.sin(lon), 0.0, None)[None, :]
        flux *= rng.uniform(0.9, 1.0, size=flux.shape)   # rough ground: partly shadowed cells
        return {"case": case, "ctx": D.Context(0), "tp": tp, "flux": flux}
    spot, facet = W.cratered_mesh(case["nlevel"], craters=24, depth=0.2, width=0.2,
                                  seed=int(rng.integers(0, 2**31)))
    return {"case": case, "ctx": D.Context(0), "spot": spot, "facet": facet,
            "normal": N.mesh_normals(spot, facet)["normal"], "za": float(rng.uniform(0.05, 0.5))}


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "solve":
        return state["ctx"].solve(PATHS[case["path"]], state["params"], state["surface"], case["n"],
                                  outputs=case["rows"])
    if kind == "reference":
        ctx = state["ctx"]
        out = ctx.solve(PATHS[case["path"]], state["params"], state["surface"], case["n"], outputs=True)
        v, td, fd, ht = ctx.velocity_record(case["n"])
        # the runner's record buffer: its length does not depend on the run
        record = np.zeros((100 * 36 * 100, 6))
        record[:len(td), :3] = v
        record[:len(td), 3:] = np.stack([td, fd, ht], 1)
        out["record"] = record
        out["n_record"] = len(td)
        return out
    if kind == "advanced":
        ctx = state["ctx"]
        fits = ctx.fit_samples(state["speeds"], state["counts"], 3)
        col = N.CollisionInputs(state["n_bg"], *fits, 3)
        out = ctx.solve(PATHS[case["path"]], state["params"], state["surface"], case["n"],
                        collision=col, outputs=True)
        out["fits"] = fits
        return out
    if kind == "two_phase":
        R, GM = W.BODIES["ceres"]
        P = W.collisional_problem(state["ctx"], "two-phase", R, GM, 50, state["seed"], state["sun"],
                                  state["T_ss"], case["n1"], case["n2"])
        out = state["ctx"].solve(N.PATH_FAST_FP32, P.params, P.surface, P.n, collision=P.collision)
        c = P.collision
        out["tables"] = [c.n_bg, c.coef, c.box, c.total, c.valid]
        return out
    if kind == "batch":
        srv = state["server"]
        tickets = [srv.submit(q.params, q.surface, q.n) for q in state["problems"]]
        done = srv.run_all(tickets)
        return [np.concatenate([done[t]["density"].ravel() for t in tickets]),
                np.concatenate([done[t]["horizon"].ravel() for t in tickets]),
                np.array([list(done[t]["stats"].values()) for t in tickets])]
    if kind == "thermal":
        return state["ctx"].thermal(case["ftd"], case["ffd"], state["tp"], state["flux"])
    return state["ctx"].shadow_flux(state["spot"], state["facet"], state["normal"], state["za"],
                                    case["tt"], case["nmonte"])


# ------------------------------------------------------------------------------------------


def _thermal_shape(case):
    dt = 9.07417 * 3600.0 / case["ffd"] / case["n_substep"]
    dr = math.sqrt(0.1 * 2.0 * dt * 6e-4 / 730.0 / 1300.0)
    return dt, dr, max(3, math.ceil(0.05 / dr))


def work(case):
    kind = case["kind"]
    grid = 36 * 72 * 8
    if kind == "solve":
        steps = case["n"] * LIFE_STEPS[case["body"]]
        rows = case["n"] * 84 if case["rows"] else 0
        return {"bytes": (case["hd"] + 1) * grid + 1280 * 80 + rows, "flops": FLOPS_PER_STEP * steps}
    if kind in ("reference", "advanced"):
        hd = 100 if kind == "reference" else 50
        fits = 36 * 72 * 50 * (50 + 13) * 8 if kind == "advanced" else 0
        return {"bytes": (hd + 2) * grid + case["n"] * 84 + fits,
                "flops": FLOPS_PER_STEP * case["n"] * LIFE_STEPS[kind]}
    if kind == "two_phase":
        # both grids, the histograms of 64 bins per cell out and in, the fits out and in
        ncell = 50 * 36 * 72
        return {"bytes": ncell * 8 * (2 + 2 * 64 + 2 * 14),
                "flops": FLOPS_PER_STEP * (case["n1"] + case["n2"]) * LIFE_STEPS["ceres"]}
    if kind == "batch":
        # lognormal sizes, median 3e5, sigma 1.17; the three bodies in equal shares
        mean = 3e5 * math.exp(0.5 * 1.17 * 1.17)
        steps = sum(LIFE_STEPS[b] for b in W.BODIES) / 3.0
        return {"bytes": case["count"] * (41 * grid + 1280 * 80),
                "flops": int(FLOPS_PER_STEP * case["count"] * mean * steps)}
    if kind == "thermal":
        ncol = case["ftd"] * case["ffd"]
        h = _thermal_shape(case)[2]
        # per depth and step: right-hand side, forward and backward sweep; ~18 balance evaluations
        return {"bytes": ncol * 16, "flops": ncol * case["n_substep"] * (h * 10 + 18 * 40)}
    nface = 20 * 4 ** case["nlevel"]
    rays = nface * case["tt"] * case["nmonte"] // 2   # half of the faces are lit
    # a ray cannot do without drawing its point and one triangle test
    return {"bytes": nface * (12 + 24 + 12) + nface * case["tt"] * 8, "flops": rays * 60}


def exact(case, seed):
    """The thermal model in 64 bits; the other outputs are whole numbers, or follow particles or
    rays through so many steps and candidates that they have no quick independent value."""
    if case["kind"] != "thermal":
        return None
    state = prepare(case, seed)
    tp, F = state["tp"], np.abs(state["flux"]).ravel()
    dt, dr, h = _thermal_shape(case)
    R = tp.conductivity * dt / tp.density / 2.0 / tp.Cp / (dr * dr)
    kdr = tp.conductivity / dr
    p, L = list(tp.p_mat), list(tp.LH_mat)

    def balance(T, below):
        lg = np.log10(T)
        pres = tp.tran_unit_p * 10.0 ** (p[0] / T + p[1] + p[2] * T + p[3] * T * T + p[4] * lg)
        heat = tp.tran_unit_LH * (L[0] / T + L[1] + L[2] * T + L[3] * T * T + L[4] * lg)
        loss = heat * np.sqrt(18e-3 / 6.02e23 / (2.0 * math.pi * 1.38e-23 * T)) * pres
        return F + kdr * below - kdr * T - 5.6704e-8 * T * T * T * T - loss

    x = np.tile(np.where(F > 0, (F / 5.6704e-8) ** 0.25, 100.0), (h, 1))
    for _ in range(tp.n_substep):
        below = x[1].copy()
        lo, hi = np.full_like(F, 50.0), np.full_like(F, 300.0)
        flo, fhi = balance(lo, below), balance(hi, below)
        on = np.ones(F.shape, dtype=bool)
        for _ in range(30):
            on &= hi < 10000.0
            widen = on & (flo * fhi > 0)
            halve = on & ~widen
            hi = np.where(widen, hi * 5.0, hi)
            mid = (lo + hi) / 2.0
            f = balance(np.where(widen, hi, mid), below)
            fhi = np.where(widen, f, fhi)
            up = halve & (flo * f <= 0)
            down = halve & ~up
            hi, fhi = np.where(up, mid, hi), np.where(up, f, fhi)
            lo, flo = np.where(down, mid, lo), np.where(down, f, flo)
            on &= ~(halve & (np.abs(lo - hi) <= 0.01))
        x[0] = (lo + hi) / 2.0
        rhs = np.zeros_like(x)
        rhs[0] = x[0]
        rhs[1:-1] = R * x[:-2] + (1.0 - 2.0 * R) * x[1:-1] + R * x[2:]
        cp, dp = np.zeros(h), np.zeros_like(x)
        dp[0] = rhs[0]
        for i in range(1, h):
            a, b, c = (-R, 1.0 + 2.0 * R, -R) if i < h - 1 else (-1.0 / dr, 1.0 / dr, 0.0)
            piv = b - a * cp[i - 1]
            cp[i] = c / piv
            dp[i] = (rhs[i] - a * dp[i - 1]) / piv
        x[-1] = dp[-1]
        for i in range(h - 2, -1, -1):
            x[i] = dp[i] - cp[i] * x[i + 1]
    return x[0].reshape(case["ftd"], case["ffd"]), None
