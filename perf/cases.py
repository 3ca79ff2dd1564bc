"""The work that a user of this framework has it do, as cases that can be timed.

A case is one whole simulation call through the Python host mirror: the trajectories of a batch of
problems are integrated (``SimulationGPU.MainLoop``) and the distributions that the problems bin, or the
final states of the trajectories, are read back. The set-ups are those of ``spectrum_gb300.workloads``
(the benchmark's families and the test suite's sizes), in both arithmetics: the FP64 drop-in, which is the
library's default, and the batched FP32 stepper. A user's program keeps its context, so ``prepare`` opens
it and ``run`` continues the job: each pass draws the next trajectory ids and adds to the same
distributions. The ``oneshot`` cases make the whole call instead, from the problem to the results.

Times of flight are shortened where a whole trajectory would take seconds (a modulation trajectory ends
after ~1e5 steps, a drift around the Earth after ~1e7): a pass stays well below two seconds.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from spectrum_gb300 import capi, workloads
from spectrum_gb300 import units as U
from spectrum_gb300.problem import Grid
from spectrum_gb300.simulation import open_problems, run_problems

PREC = {"fp64": capi.SPX_FP64, "mixed": capi.SPX_MIXED}


def listed():
    return [
        # the smallest call: a smoke test or one point of a scripted scan, from the problem to its
        # histogram; latency, allocations and launches count
        {"name": "diffusion_fp64_oneshot", "family": "diffusion", "prec": "fp64", "oneshot": True, "n_traj": 64,
         "t_end": 0.05, "kappa": 1.0, "n_bins": 100, "record": True},
        # pure diffusion as the reference's benchmark has it: 1e5 trajectories, dt = 1e-3 to t = 1, 100^3 bins
        {"name": "diffusion_fp64", "family": "diffusion", "prec": "fp64", "oneshot": False, "n_traj": 100_000,
         "t_end": 1.0, "kappa": 1.0, "n_bins": 100, "record": False},
        # the same in the batched stepper at the benchmark's 1e6
        {"name": "diffusion_mixed", "family": "diffusion", "prec": "mixed", "oneshot": False, "n_traj": 1_000_000,
         "t_end": 1.0, "kappa": 1.0, "n_bins": 100, "record": False},
        # diffusive shock acceleration: planes and a momentum boundary, run time of a trajectory very uneven
        {"name": "shock_mixed", "family": "shock", "prec": "mixed", "oneshot": False, "n_traj": 40_000, "width": 0.03,
         "half": 2.0, "p_max": 20.0, "record": False},
        # full orbits in the dipole, the batched stepper and the drop-in (final states, as the drift-period
        # and energy-drift comparisons read them)
        {"name": "dipole_mixed", "family": "dipole", "prec": "mixed", "oneshot": False, "n_traj": 200_000, "t_end_s": 1.0,
         "record": False},
        {"name": "dipole_fp64", "family": "dipole", "prec": "fp64", "oneshot": False, "n_traj": 4001, "t_end_s": 0.25,
         "record": True},
        # cosmic-ray modulation in the Parker spiral, backward in time: the headline workload. Batched, and
        # the drop-in with the reference's numerical derivatives at a test-like size
        {"name": "modulation_mixed", "family": "modulation", "prec": "mixed", "oneshot": False, "n_traj": 6000,
         "n_energies": 32, "t_max_years": 0.1, "pow_law_b": -1.0, "record": False},
        {"name": "modulation_fp64", "family": "modulation", "prec": "fp64", "oneshot": False, "n_traj": 300,
         "n_energies": 4, "t_max_years": 0.005, "pow_law_b": 0.0, "record": False},
        # focused transport with scattering: many problems of ragged sizes in one launch
        {"name": "focused_mixed", "family": "focused", "prec": "mixed", "oneshot": False, "n_problems": 64, "n_min": 100,
         "n_max": 4000, "t_max_hours": 0.25, "record": False},
        # trapped protons as guiding centres, with mirror-point events
        {"name": "guiding_mixed", "family": "guiding", "prec": "mixed", "oneshot": False, "n_traj": 100_000, "t_end_s": 10.0,
         "record": False},
        {"name": "guiding_fp64", "family": "guiding", "prec": "fp64", "oneshot": False, "n_traj": 512, "t_end_s": 10.0,
         "record": True},
        # modulation on a gridded background of 256^3 nodes (537 MB of node data: past the L2)
        {"name": "grid_mixed", "family": "grid", "prec": "mixed", "oneshot": False, "n_traj": 10_000, "n_energies": 8,
         "n_nodes": 256, "t_max_years": 0.2, "record": False},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random):
    """One more case of the ranges the listed ones stand for (sizes log-uniform, odd ones among them)."""
    family, prec = rng.choice([("diffusion", "fp64"), ("diffusion", "mixed"), ("shock", "mixed"), ("dipole", "mixed"),
                               ("dipole", "fp64"), ("modulation", "mixed"), ("modulation", "fp64"), ("focused", "mixed"),
                               ("guiding", "mixed"), ("guiding", "fp64"), ("grid", "mixed")])
    fp64 = prec == "fp64"
    c = {"family": family, "prec": prec, "oneshot": rng.random() < 0.2, "record": False}
    if family == "diffusion":
        c.update(n_traj=int(_log(rng, 50, 100_000 if fp64 else 1_000_000)), t_end=round(_log(rng, 0.05, 1.0), 4),
                 kappa=round(_log(rng, 0.5, 2.0), 3), n_bins=rng.randint(20, 100), record=rng.random() < 0.3)
        if c["n_traj"] > 100_000:
            c["record"] = False
    elif family == "shock":
        c.update(n_traj=int(_log(rng, 500, 40_000)), width=round(_log(rng, 0.03, 0.1), 4),
                 half=round(rng.uniform(1.0, 2.0), 3), p_max=round(_log(rng, 5.0, 20.0), 2))
    elif family == "dipole":
        if fp64:
            c.update(n_traj=int(_log(rng, 50, 4001)), t_end_s=round(_log(rng, 0.05, 0.25), 4), record=rng.random() < 0.7)
        else:
            c.update(n_traj=int(_log(rng, 500, 200_000)), t_end_s=round(_log(rng, 0.1, 1.0), 4))
    elif family == "modulation":
        if fp64:
            c.update(n_traj=int(_log(rng, 16, 300)), n_energies=rng.randint(1, 4),
                     t_max_years=round(_log(rng, 0.001, 0.005), 5), pow_law_b=rng.choice([0.0, -1.0]))
        else:
            c.update(n_traj=int(_log(rng, 50, 6000)), n_energies=rng.randint(1, 32),
                     t_max_years=round(_log(rng, 0.02, 0.1), 5), pow_law_b=rng.choice([0.0, -1.0]))
    elif family == "focused":
        c.update(n_problems=rng.randint(1, 64), n_min=100, n_max=int(_log(rng, 200, 4000)),
                 t_max_hours=round(_log(rng, 0.02, 0.25), 4))
    elif family == "guiding":
        if fp64:
            c.update(n_traj=int(_log(rng, 50, 512)), t_end_s=round(_log(rng, 1.0, 10.0), 3), record=rng.random() < 0.7)
        else:
            c.update(n_traj=int(_log(rng, 500, 100_000)), t_end_s=round(_log(rng, 1.0, 10.0), 3))
    else:
        c.update(n_traj=int(_log(rng, 100, 10_000)), n_energies=rng.randint(1, 8), n_nodes=rng.choice([64, 96, 128, 256]),
                 t_max_years=round(_log(rng, 0.02, 0.2), 5))
    return c


# -- set-up ------------------------------------------------------------------------------------------
def _seed(seed):
    return (0x9E3779B97F4A7C15 * (int(seed) + 1)) & 0xFFFFFFFFFFFFFFFF


def _spiral_grid(n, half_width_au):
    """The Parker spiral on n^3 nodes, as workloads.gcr_modulation_grid samples it, evaluated on the GPU:
    the numbers that a user's program has read from a file."""
    h = half_width_au * workloads.ONE_AU
    zone = 2.0 * h / (n - 1)
    ax = -h + zone * torch.arange(n, dtype=torch.float64, device="cuda")
    z, y, x = torch.meshgrid(ax, ax, ax, indexing="ij")
    umag = 4.0e7 / U.unit_velocity
    r_ref = 3.0 * 6.957e10 / U.unit_length
    a = (5.0e-5 / U.unit_magnetic) * (workloads.ONE_AU / r_ref) ** 2 * r_ref * r_ref
    k = a * (2.0 * math.pi / (25.0 * 24.0 * 3600.0) * U.unit_time) / umag
    r = torch.sqrt(x * x + y * y + z * z)
    ur, ar, f = umag / r, a / r ** 3, k * (r - r_ref) / r ** 3
    v = torch.stack([ur * x, ur * y, ur * z, ar * x + f * y, ar * y - f * x, ar * z], dim=-1)
    return Grid((n,) * 3, (-h,) * 3, (zone,) * 3, v.cpu().numpy())


def _problems(case, seed):
    f = case["family"]
    if f == "diffusion":
        pbs = [workloads.diffusion_uniform(n_traj=case["n_traj"], t_end=case["t_end"], kappa=case["kappa"],
                                           n_bins=case["n_bins"])]
    elif f == "shock":
        pbs = [workloads.shock_acceleration(n_traj=case["n_traj"], width_frac=case["width"], x_escape=-case["half"],
                                            x_downstream=case["half"], p_max=case["p_max"])]
    elif f == "dipole":
        pbs = [workloads.dipole_orbits(n_traj=case["n_traj"], t_end=case["t_end_s"] / U.unit_time)]
    elif f == "modulation":
        pbs = workloads.gcr_modulation(n_traj=case["n_traj"], energies_mev=workloads.modulation_energies(case["n_energies"]),
                                       t_max_years=case["t_max_years"], pow_law_b=case["pow_law_b"])
    elif f == "focused":
        pbs = workloads.focused_transport(n_problems=case["n_problems"], n_min=case["n_min"], n_max=case["n_max"],
                                          t_max_hours=case["t_max_hours"])
    elif f == "guiding":
        pbs = [workloads.guiding_dipole(n_traj=case["n_traj"], t_end_s=case["t_end_s"])]
    else:
        # a few nodes make the set-up, then the block of this case takes their place
        pbs = workloads.gcr_modulation_grid(n_traj=case["n_traj"], n_nodes=4, t_max_years=case["t_max_years"],
                                            energies_mev=workloads.modulation_energies(case["n_energies"], 30.0, 3.0e3))
        grid = _spiral_grid(case["n_nodes"], 6.0)
        for p in pbs:
            p.grid = grid
    for p in pbs:
        p.seed = _seed(seed)
    return pbs


def prepare(case, seed):
    pbs = _problems(case, seed)
    s = {"case": case, "problems": pbs, "prec": PREC[case["prec"]], "n_distros": len(pbs[0].distributions())}
    if not case["oneshot"]:
        s["sim"] = open_problems(pbs, precision=s["prec"], record=case["record"])
    return s


# -- one pass ------------------------------------------------------------------------------------------
def _outputs(stats, distros, records):
    """The distributions of all problems, end to end, and the final states when the run keeps them."""
    out = {"trajectories": stats.trajectories, "steps": stats.steps, "given_up": stats.given_up, "events": stats.events,
           "counts": np.concatenate([d[0] for d in distros]), "sums": np.concatenate([d[1].ravel() for d in distros]),
           "n_events": np.array([d[2] for d in distros], dtype=np.int64)}
    if records:
        r = np.concatenate(records)
        out.update(rec_status=r["status"].astype(np.int64), rec_steps=r["steps"].astype(np.int64), rec_t=r["t"].copy(),
                   rec_pos=r["pos"].copy(), rec_mom=r["mom"].copy())
    return out


def run(s):
    pbs, record = s["problems"], s["case"]["record"]
    if s["case"]["oneshot"]:
        res = run_problems(pbs, precision=s["prec"], record=record)
        return _outputs(res.stats, [d for p in res.distros for d in p], res.records)
    sim = s["sim"]
    stats = sim.MainLoop()
    distros = [sim.distribution(d, k) for k in range(len(pbs)) for d in range(s["n_distros"])]
    records = [sim.ctx.records(k, p.n_traj) for k, p in enumerate(pbs)] if record else None
    return _outputs(stats, distros, records)


# Operations of one accepted step with analytic field derivatives (additions and multiplications, as the
# repository's op-counting oracle counts them) and a typical number of steps of a trajectory, measured on
# these set-ups: a step reads and writes nothing in memory but the nodes of a gridded background.
FLOP = {"diffusion": 15.0, "shock": 60.0, "dipole": 400.0, "modulation": 350.0, "focused": 450.0, "guiding": 600.0,
        "grid": 600.0}


def _steps(case):
    f = case["family"]
    if f == "diffusion":
        return case["t_end"] * 1000.0  # dt = 1e-3 whatever kappa is
    if f == "shock":
        return 3.3e4 * (0.03 / case["width"]) * (case["half"] / 2.0)
    if f == "dipole":
        return 1075.0 * case["t_end_s"]
    if f == "modulation":
        return 2.0e5 * case["t_max_years"]
    if f == "focused":
        return 3.4e4 * case["t_max_hours"]
    if f == "guiding":
        return 143.0 * case["t_end_s"]
    return 8.5e4 * case["t_max_years"]


def _total(case):
    if case["family"] == "focused":
        return case["n_problems"] * (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
    return case["n_traj"] * case.get("n_energies", 1)


def work(case):
    n = _total(case)
    bins = {"diffusion": case.get("n_bins", 0) ** 3, "shock": 200, "dipole": 2048, "guiding": 2108,
            "modulation": case.get("n_energies", 0) * (4 * case.get("n_energies", 0) + 32),
            "grid": case.get("n_energies", 0) * (4 * case.get("n_energies", 0) + 32),
            "focused": case.get("n_problems", 0) * 8192}[case["family"]]
    nbytes = 12.0 * bins + (144.0 * n if case["record"] else 0.0)
    if case["family"] == "grid":
        nbytes += 28.0 * case["n_nodes"] ** 3
    return {"bytes": nbytes, "flops": n * _steps(case) * FLOP[case["family"]]}


# -- the same numbers in plain 64-bit torch ----------------------------------------------------------------
def _mulhilo(a, b):
    """High and low 32 bits of a * b: b a constant, both below 2^32, in int64."""
    p0, p1 = a * (b & 0xFFFF), a * (b >> 16)
    lo = p0 + ((p1 & 0xFFFF) << 16)
    return (p1 >> 16) + (lo >> 32), lo & 0xFFFFFFFF


def _philox(c, key):
    """Philox4x32-10 of Salmon, Moraes, Dror and Shaw (SC'11) on four int64 tensors of 32-bit words."""
    k0, k1 = key & 0xFFFFFFFF, key >> 32
    for _ in range(10):
        h0, l0 = _mulhilo(c[0], 0xD2511F53)
        h1, l1 = _mulhilo(c[2], 0xCD9E8D57)
        c = (h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0)
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _uniforms(seed, index, traj, purpose):
    i = torch.full_like(traj, index)
    c = _philox((i, traj, torch.zeros_like(traj), torch.full_like(traj, purpose << 24)), _seed(seed))
    return [(x.double() + 0.5) * 2.0 ** -32 for x in c]


def _binned(cols, lo, width, n):
    """Counts of one event per row, linear index with the last column fastest; the caller drops outliers."""
    idx = torch.zeros_like(cols[0], dtype=torch.int64)
    for x, a, w, m in zip(cols, lo, width, n):
        idx = idx * m + ((x - a) / w).long().clamp(0, m - 1)
    return torch.bincount(idx, minlength=int(np.prod(n))).double()


def _floats(sums, rec=None):
    """The layout of ``_outputs``: only its computed numbers have a value here."""
    out = dict.fromkeys(("trajectories", "steps", "given_up", "events", "counts", "n_events"))
    out["sums"] = sums.cpu().numpy()
    if rec is not None:
        out.update(rec_status=None, rec_steps=None, **{k: v.cpu().numpy() for k, v in rec.items()})
    return out


def _exact_diffusion(case, seed):
    """Every trajectory takes the same steps: dt = 1e-3, the last one just past t_end; B along z."""
    n, kappa, t_end, nb = case["n_traj"], case["kappa"], case["t_end"], case["n_bins"]
    c_light = U.c_code
    dmax = math.sqrt(2.0 * kappa * 1.0e-3)
    dt0 = 0.5 * dmax * dmax / kappa
    traj = torch.arange(n, dtype=torch.int64, device="cuda")
    pos = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
    s, t, k = math.sqrt(2.0 * kappa), 0.0, 0
    while t - t_end < 0.0:
        left = t_end - t
        dt = max((1.0 + 1.0e-5) * left, 1.0e-8 * dmax / c_light) if dt0 >= left else dt0
        u = _uniforms(seed, k, traj, 0)
        r0, r1 = torch.sqrt(-2.0 * torch.log(u[0])), torch.sqrt(-2.0 * torch.log(u[2]))
        a0, a1 = 2.0 * math.pi * u[1], 2.0 * math.pi * u[3]
        d = torch.stack([-r0 * torch.cos(a0), -r0 * torch.sin(a0), r1 * torch.cos(a1)], dim=1)
        pos += s * math.sqrt(dt) * d
        t, k = t + dt, k + 1
    inside = ((pos >= -6.0) & (pos < 6.0)).all(dim=1)
    p = pos[inside]
    sums = _binned([p[:, 0], p[:, 1], p[:, 2]], (-6.0,) * 3, (12.0 / nb,) * 3, (nb,) * 3)
    rec = None
    if case["record"]:
        mom = torch.zeros_like(pos)
        mom[:, 0] = 1.0
        rec = {"rec_t": torch.full((n,), t, dtype=torch.float64), "rec_pos": pos, "rec_mom": mom}
    return _floats(sums, rec)


def _exact_dipole(case, seed):
    """Newton-Lorentz orbits of protons in the dipole, classic fourth-order Runge-Kutta, 32 steps a gyration."""
    n, c = case["n_traj"], U.c_code
    traj = torch.arange(n, dtype=torch.int64, device="cuda")
    r_e, b_eq = workloads.R_EARTH_CM / U.unit_length, workloads.B_EARTH_G / U.unit_magnetic
    t_end = case["t_end_s"] / U.unit_time
    m = torch.tensor([0.0, 0.0, -b_eq * r_e ** 3], dtype=torch.float64, device="cuda")

    def norm(v):
        return torch.sqrt((v * v).sum(dim=1))

    def field(x):
        r2 = (x * x).sum(dim=1, keepdim=True)
        return (3.0 * (x @ m)[:, None] * x - r2 * m) / (r2 * r2 * torch.sqrt(r2))

    def velocity(p):
        return p * (c / torch.sqrt((p * p).sum(dim=1, keepdim=True) + c * c))

    # initial conditions: uniforms 0, 1 the L shell and azimuth; the momentum is drawn twice (before and after
    # the field at the start is known), so uniforms 5, 6, 7 are the energy, pitch cosine and gyrophase
    u = [_uniforms(seed, b, traj, 1)[i] for b, i in ((0, 0), (0, 1), (1, 1), (1, 2), (1, 3))]
    ell, phi = 2.0 + 4.0 * u[0], 2.0 * math.pi * u[1]
    x = torch.stack([ell * r_e * torch.cos(phi), ell * r_e * torch.sin(phi), torch.zeros_like(phi)], dim=1)
    e1, e2 = math.log(U.MEV / U.unit_energy), math.log(100.0 * U.MEV / U.unit_energy)
    e = torch.exp(e1 + (e2 - e1) * u[2])
    mu_lo, mu_hi = math.cos(math.radians(170.0)), math.cos(math.radians(10.0))
    mu, psi = mu_lo + (mu_hi - mu_lo) * u[3], 2.0 * math.pi * u[4]
    p_abs = torch.sqrt(e * (e + 2.0 * c * c)) / c
    b = field(x)
    bh = b / norm(b)[:, None]
    # the first perpendicular vector: b x the axis of its smallest component (y, then z where two are equal)
    ax, ay, az = bh.abs().unbind(dim=1)
    least = torch.where(ax < ay, torch.where(ax < az, 0, 2), torch.where(ay < az, 1, 2))
    e_min = torch.nn.functional.one_hot(least, 3).double()
    w1 = torch.linalg.cross(bh, e_min)
    w1 = w1 / norm(w1)[:, None]
    w2 = torch.linalg.cross(bh, w1)
    st = torch.sqrt(1.0 - mu * mu)
    p = (p_abs * mu)[:, None] * bh + (p_abs * st)[:, None] * (torch.cos(psi)[:, None] * w1 + torch.sin(psi)[:, None] * w2)
    t = torch.zeros(n, dtype=torch.float64, device="cuda")
    alive = torch.arange(n, device="cuda")
    while alive.numel():
        xa, pa, ta = x[alive], p[alive], t[alive]
        v0, b0 = velocity(pa), field(xa)
        vn, bm, r = norm(v0), norm(b0), norm(xa)
        gyro = bm / (c / torch.sqrt(1.0 - (vn / c) ** 2))
        dmax = (0.1 * r).clamp(max=0.1 * r_e)
        dt = torch.minimum(2.0 * math.pi / gyro / 32.0, 0.1 * dmax / vn)
        left = t_end - ta
        dt = torch.where(dt >= left, torch.maximum((1.0 + 1.0e-5) * left, 1.0e-8 * dmax / c), dt)[:, None]
        k = [(v0, torch.linalg.cross(v0, b0) / c)]
        hit = torch.zeros_like(alive, dtype=torch.bool)
        xs, ps = xa, pa
        for stage, h in ((1, 0.5), (2, 0.5), (3, 1.0)):
            xs, ps = torch.where(hit[:, None], xs, xa + h * dt * k[-1][0]), torch.where(hit[:, None], ps, pa + h * dt * k[-1][1])
            # the reference advances a stage's time once for every earlier stage (src/trajectory_base.cc:329-337)
            ta = torch.where(hit, ta, t[alive] + stage * h * dt[:, 0])
            hit = hit | (norm(xs) <= r_e)
            v = velocity(ps)
            k.append((v, torch.linalg.cross(v, field(xs)) / c))
        w = (1.0 / 6.0, 1.0 / 3.0, 1.0 / 3.0, 1.0 / 6.0)
        xn = xa + dt * sum(a * q[0] for a, q in zip(w, k))
        pn = pa + dt * sum(a * q[1] for a, q in zip(w, k))
        # a stage point inside the Earth ends the trajectory there
        x[alive] = torch.where(hit[:, None], xs, xn)
        p[alive] = torch.where(hit[:, None], ps, pn)
        t[alive] = torch.where(hit, ta, t[alive] + dt[:, 0])
        done = hit | (norm(x[alive]) <= r_e) | (t[alive] >= t_end)
        alive = alive[~done]
    rec = {"rec_t": t, "rec_pos": x, "rec_mom": p} if case["record"] else None
    # the histogram bins the pitch cosine against the field of the last stage point; a few orbits end on a
    # bin's edge, so it has no value to hold the sums to
    out = _floats(torch.zeros(1), rec)
    out["sums"] = None
    return out


def exact(case, seed):
    """Plain torch in 64 bits for pure diffusion and for the dipole's orbits with final states. The other
    families have none: their paths are chaotic (a change of the last bit moves them by more than any bound)
    and a pass makes 1e8 to 1e10 steps, which torch cannot take in 20 seconds."""
    if case["family"] == "diffusion" and case["n_traj"] * case["t_end"] <= 1.1e6:
        return _exact_diffusion(case, seed)
    if case["family"] == "dipole" and case["prec"] == "fp64" and case["record"]:
        return _exact_dipole(case, seed)
    return None
