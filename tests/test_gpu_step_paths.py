"""The step's special paths against the general ones: what a path takes over gives the same trajectories.

- Quotients by a shared divisor leave their fast form where an exponent could over- or underflow: a dmax of
  1e140 takes the time-step bounds there (FP64 against the oracle).
- Stage points told by their clearance from the boundaries, against the oracle's evaluation of each; steps so small
  that the positions' rounding is a part of the way, against the step count that arithmetic gives.
- The FP32 kernels compiled for a boundary layout against the one that reads it from the descriptor.
- The deep build of the FP32 kernels, with its repacking of lanes, against the wide one.
- The initial momentum, of whose two samples the first is only counted where nothing reads it, against the oracle.
- Small FP64 launches: teams of lanes sharing a trajectory against one lane each.
- Steps that cross two reflecting boundaries, against the oracle.
- Launches of few trajectories keep their shape when the autotuner has run or when a run is given back what another
  reported; larger ones take the tuned shape.
- Uniform fields: coefficients held over a trajectory (diffusion classes that do not read the position)
  and evaluated at every step (those that do), in both time flows: FP64 against the oracle, and the FP32
  kernels of one diffusion class against the kernel that dispatches at run time, whose steps are general."""
import numpy as np
import pytest

import oracle_tools as ot
import test_oracle_plugins as cases
from spectrum_gb300 import capi, units
from spectrum_gb300 import plugins as P
from spectrum_gb300 import workloads as W
from spectrum_gb300.datacontainer import DataContainer as DC
from spectrum_gb300.plugins import (BoundaryPlaneAbsorb, BoundaryPlaneReflect, DiffusionRigidityMagneticFieldPowerLaw,
                                    InitialMomentumLogEnergyPitchBand)
from spectrum_gb300.simulation import open_problems, run_problems

pytestmark = pytest.mark.gpu

UNIFORM_DIFFUSION = {
    "full": (cases.DiffusionFullConstant(), DC().double(0.5).double(2.0)),
    "rigidity_b": (DiffusionRigidityMagneticFieldPowerLaw(),
                   DC().double(0.3).double(5.0).double(0.7).double(0.5).double(1.0).double(0.1)),
    "radial": cases.DIFFUSION_CASES["kin_energy_radial"][0],  # reads the position: the general step
}


def _uniform(name, flow, n):
    bg = (cases.BackgroundUniform(), DC().double(0.0).vec((0, 0, 0)).vec((0.2, 0.1, -0.1)).vec((0.3, -0.2, 0.8)).double(0.05))
    return cases._parker(n=n, bg=bg, diff=UNIFORM_DIFFUSION[name], flow=flow, t_end=0.1 if flow == cases.FORWARD else -0.1,
                         is_=(cases.InitialSpaceFixed(), DC().vec((0.3, 0, 0))),
                         bnds=[(cases.BoundarySphereReflect(), cases.B(DC(), -1, [-1]).vec((0, 0, 0)).double(0.6))])


@pytest.mark.parametrize("flow", [cases.FORWARD, cases.BACKWARD])
@pytest.mark.parametrize("name", sorted(UNIFORM_DIFFUSION))
def test_uniform_field_matches_oracle(built_lib, name, flow):
    pb = _uniform(name, flow, 33)
    res = run_problems(pb, precision=capi.SPX_FP64, record=True)
    ot.assert_fp64_parity(res.records[0], ot.run_oracle(pb), ot.run_oracle(pb, nudge_libm=1), distros=res.distros[0])


@pytest.mark.parametrize("flow", [cases.FORWARD, cases.BACKWARD])
@pytest.mark.parametrize("name", ["full", "rigidity_b"])
def test_uniform_field_fp32_equals_the_general_step(built_lib, name, flow):
    rec = []
    for special in (0, 1):
        sim = open_problems(_uniform(name, flow, 1000), precision=capi.SPX_MIXED, record=True)
        sim.ctx.set_option(capi.SPX_OPT_SPECIALIZE, float(special))
        sim.MainLoop()
        rec.append(sim.ctx.records(0, 1000))
        sim.close()
    for f in ("status", "steps", "t", "pos", "mom"):
        assert np.array_equal(rec[0][f], rec[1][f]), f


def test_quotients_outside_the_fast_range(built_lib):
    bg = (cases.BackgroundUniform(), DC().double(0.0).vec((0, 0, 0)).vec((0, 0, 0)).vec((0, 0, 1.0)).double(1.0e140))
    pb = cases._parker(n=40, bg=bg, t_end=0.1)
    res = run_problems(pb, precision=capi.SPX_FP64, record=True)
    ot.assert_fp64_parity(res.records[0], ot.run_oracle(pb), ot.run_oracle(pb, nudge_libm=1), distros=res.distros[0])


@pytest.mark.parametrize("n", [1, 31, 700, 2433, 4865, 9729])
@pytest.mark.parametrize("kind", ["modulation", "focused", "guiding", "lorentz"])
def test_lane_teams_equal_single_lanes(built_lib, kind, n):
    """Small FP64 launches give a trajectory several lanes (eight up to 2,432 trajectories, four, two, then one) and
    spread over all schedulers; the launch shape given here has one lane each in full warps."""
    if kind == "modulation":
        pb = W.gcr_modulation(n_traj=n, energies_mev=[300.0], t_max_years=1.0e-4, pow_law_b=-1.0)[0]
    elif kind == "focused":
        pb = W.focused_transport(n_problems=1, n_traj=n, t_max_hours=0.002)[0]
    elif kind == "guiding":
        pb = W.guiding_dipole(n_traj=n, t_end_s=0.1)
    else:
        pb = W.dipole_orbits(n_traj=n, t_end=0.01 / units.unit_time)
    a = run_problems(pb, precision=capi.SPX_FP64, record=True)
    b = run_problems(pb, precision=capi.SPX_FP64, record=True, tuning=capi.Tuning(128, 0, 0, 0))
    assert a.stats.trajectories == b.stats.trajectories == n and a.stats.steps == b.stats.steps > n
    assert a.stats.events == b.stats.events
    for f in ("attempts", "status", "steps", "t", "pos", "mom"):
        assert np.array_equal(a.records[0][f], b.records[0][f]), f
    for (ca, _, na), (cb, _, nb) in zip(a.distros[0], b.distros[0]):
        assert na == nb and np.array_equal(ca, cb)


@pytest.mark.parametrize("n", [1, 33, 129, 4097, 60_001])
@pytest.mark.parametrize("kind", ["uniform", "spiral", "shock", "grid", "dipole"])
def test_deep_build_equals_the_wide_one(built_lib, kind, n):
    """Untuned FP32 runs of few trajectories a lane take the kernels' deep build, whose blocks repack their lanes as
    trajectories end; a given launch shape takes the wide build. The same trajectories, bit for bit."""
    if kind == "uniform":
        pbs = [W.diffusion_uniform(n_traj=min(n, 50_000), t_end=0.02)]
    elif kind == "spiral":  # two problems of different length, retries and both exits
        pbs = W.gcr_modulation(n_traj=(n + 1) // 2, energies_mev=[30.0, 1000.0], t_max_years=0.005, pow_law_b=-1.0)
    elif kind == "shock":
        pbs = [W.shock_acceleration(n_traj=n, width_frac=0.2, x_escape=-0.3, x_downstream=0.3, p_max=2.0)]
    elif kind == "grid":
        pbs = W.gcr_modulation_grid(n_traj=n, n_nodes=32, energies_mev=[300.0], t_max_years=0.005)
    else:
        pbs = [W.dipole_orbits(n_traj=n, t_end=0.05 / units.unit_time)]
    a = run_problems(pbs, precision=capi.SPX_MIXED, record=True)
    b = run_problems(pbs, precision=capi.SPX_MIXED, record=True, tuning=capi.Tuning(64, 0, 8, 1))
    assert a.stats.tuning.block_size == 128 and a.stats.steps == b.stats.steps and a.stats.retries == b.stats.retries
    for ra, rb in zip(a.records, b.records):
        for f in ("attempts", "status", "steps", "t", "pos", "mom", "pos0", "mom0"):
            assert np.array_equal(ra[f], rb[f]), f
    for da, db in zip(a.distros, b.distros):
        for (ca, _, na), (cb, _, nb) in zip(da, db):
            assert na == nb and np.array_equal(ca, cb)


@pytest.mark.parametrize("n", [1, 1000])
@pytest.mark.parametrize("kind", ["absorbing_planes", "reflecting_planes_momentum_pass", "time_only"])
def test_boundary_layout_kernels_equal_the_generic_one(built_lib, kind, n):
    """The FP32 Parker kernels compiled for two planes with a momentum boundary, and for a time boundary alone,
    against the kernel that reads kinds and counts from the descriptor: crossings of every boundary among them."""
    c = cases
    if kind == "absorbing_planes":
        pb = W.shock_acceleration(n_traj=n, width_frac=0.1, x_escape=-0.3, x_downstream=0.3, p_max=1.2)
    elif kind == "reflecting_planes_momentum_pass":
        pb = c._parker(n=n, bg=c._shock(), t_end=0.3,
                       bnds=[(BoundaryPlaneReflect(), c.B(DC(), -1, [-1]).vec((0.2, 0, 0)).vec((1.0, 0, 0))),
                             (BoundaryPlaneReflect(), c.B(DC(), -1, [-1]).vec((-0.2, 0, 0)).vec((-1.0, 0, 0))),
                             (c.BoundaryMomentumPass(), c.B(DC(), -1, [0]).double(1.01))])
    else:
        pb = W.diffusion_uniform(n_traj=n, t_end=0.1)
    out = []
    for special in (0, 1):
        sim = open_problems(pb, precision=capi.SPX_MIXED, record=True)
        sim.ctx.set_option(capi.SPX_OPT_SPECIALIZE, float(special))
        st = sim.MainLoop()
        out.append((st.events, sim.ctx.records(0, n), sim.ctx.distribution(0, 0)))
        sim.close()
    assert out[0][0] == out[1][0] and out[0][2][2] == out[1][2][2]
    for f in ("status", "steps", "t", "pos", "mom"):
        assert np.array_equal(out[0][1][f], out[1][1][f]), f
    assert np.array_equal(out[0][2][0], out[1][2][0])


@pytest.mark.parametrize("offset", [0.0, 1.0e-3, 0.05, 0.9])
@pytest.mark.parametrize("kind", ["sphere", "plane", "two_spheres_far_origin"])
def test_stage_points_near_boundaries_match_oracle(built_lib, kind, offset):
    """The clearance that stands in for the boundaries at stage points: Lorentz orbits (FP64) that start at various
    distances from an absorbing boundary, on it among them, end at the same stage or step as in the oracle."""
    c = cases
    if kind == "sphere":
        bnds = [(c.BoundarySphereAbsorb(), c.B(DC(), 1, [0]).vec((0, 0, 0)).double(1.0))]
    elif kind == "plane":
        bnds = [(BoundaryPlaneAbsorb(), c.B(DC(), 1, [0]).vec((1.0, 0, 0)).vec((1.0, 0, 0)))]
    else:
        bnds = [(c.BoundarySphereAbsorb(), c.B(DC(), 1, [0]).vec((1.0e6, 0, 0)).double(1.0e6 - 1.0)),
                (c.BoundarySphereReflect(), c.B(DC(), -1, [-1]).vec((0, 0, 0)).double(3.0))]
    bg = (c.BackgroundUniform(), DC().double(0.0).vec((0, 0, 0)).vec((0, 0, 0)).vec((0, 0.3, 1.0)).double(0.5))
    pb = c._parker(n=48, traj=c.TRAJ_LORENTZ, diff=False, bg=bg, t_end=3.0, bnds=bnds,
                   is_=(c.InitialSpaceFixed(), DC().vec((1.0 - offset, 0, 0))),
                   im=(c.InitialMomentumShell(), DC().double(0.5)))
    res = run_problems(pb, precision=capi.SPX_FP64, record=True)
    ot.assert_fp64_parity(res.records[0], ot.run_oracle(pb), ot.run_oracle(pb, nudge_libm=1), distros=res.distros[0])


@pytest.mark.parametrize("n", [1, 129, 4097, 120_001])
def test_guiding_repacking_keeps_the_orbits(built_lib, n):
    """FP32 guiding centres in blocks of 128, whose warps are repacked as orbits end, against blocks of one warp, which
    have nothing to repack: mirror-point events and final states, bit for bit."""
    pb = W.guiding_dipole(n_traj=n, t_end_s=0.5)
    a = run_problems(pb, precision=capi.SPX_MIXED, record=True)
    b = run_problems(pb, precision=capi.SPX_MIXED, record=True, tuning=capi.Tuning(32, 0, 8, 1))
    assert a.stats.tuning.block_size == 128 and a.stats.steps == b.stats.steps and a.stats.events == b.stats.events
    for f in ("attempts", "status", "steps", "t", "pos", "mom", "pos0", "mom0"):
        assert np.array_equal(a.records[0][f], b.records[0][f]), f
    for (ca, _, na), (cb, _, nb) in zip(a.distros[0], b.distros[0]):
        assert na == nb and np.array_equal(ca, cb)


INITIAL_MOMENTA = {
    "beam": (cases.InitialMomentumBeam(), DC().double(1.0)),
    "ring": (cases.InitialMomentumRing(), DC().double(1.0).double(0.7)),
    "shell": (cases.InitialMomentumShell(), DC().double(1.0)),
    "thick_shell": (cases.InitialMomentumThickShell(), DC().double(0.5).double(2.0).bool(False)),
    "thick_shell_log": (cases.InitialMomentumThickShell(), DC().double(0.5).double(2.0).bool(True)),
    "maxwell": (cases.InitialMomentumMaxwell(), DC().double(1.0).double(0.3).double(0.2)),
    "pitch_band": (InitialMomentumLogEnergyPitchBand(), DC().double(0.5).double(2.0).double(-0.5).double(0.5)),
}


@pytest.mark.parametrize("precision", [capi.SPX_FP64, capi.SPX_MIXED])
@pytest.mark.parametrize("traj,name", [
    (t, n) for t in (cases.TRAJ_PARKER, cases.TRAJ_LORENTZ, cases.TRAJ_GUIDING, cases.TRAJ_FOCUSED, cases.TRAJ_FIELDLINE)
    for n in sorted(INITIAL_MOMENTA) if n not in {cases.TRAJ_PARKER: ("beam", "ring"),
                                                  cases.TRAJ_FIELDLINE: ("beam", "ring", "pitch_band")}.get(t, ())])
def test_initial_momenta_match_oracle(built_lib, traj, name, precision):
    """A start samples its momentum twice; where the first sample is only counted, the second takes the same draws.
    FP32 kernels hold the field direction, which some samples follow, to 2**-24 per component; FP64 differs from the
    oracle by the libraries' last bits."""
    bg = (cases.BackgroundUniform(), DC().double(0.0).vec((0, 0, 0)).vec((0, 0, 0)).vec((0.3, -0.2, 0.8)).double(0.05))
    pb = cases._parker(n=70, traj=traj, bg=bg, diff=None if traj == cases.TRAJ_PARKER else False, t_end=0.01,
                       is_=(cases.InitialSpaceFixed(), DC().vec((0.1, 0.2, 0.3))), im=INITIAL_MOMENTA[name])
    rec, ref = run_problems(pb, precision=precision, record=True).records[0], ot.run_oracle(pb).traj
    scale = np.linalg.norm(ref["mom0"], axis=1, keepdims=True)
    tol = 1e-13 if precision == capi.SPX_FP64 else 1e-6
    assert np.all(np.abs(rec["mom0"] - ref["mom0"]) <= tol * scale)


@pytest.mark.parametrize("n,tuning", [(1, (64, 0, 8, 1)), (65, (64, 1, 8, 1)), (20_000, (64, 1, 8, 1)), (20_000, (64, 1, 1000, 1)),
                                      (20_000, (32, 1, 1, 1)), (20_000, (128, 1, 8, 1))])
def test_lanes_that_wait_for_a_start_change_no_orbit(built_lib, n, tuning):
    """FP32 Lorentz orbits on one block of lanes that start several orbits at a time, at most a few hundred steps late,
    against the plain grid, which has every orbit started at once: final states bit for bit."""
    pb = W.dipole_orbits(n_traj=n, t_end=0.2 / units.unit_time)
    a = run_problems(pb, precision=capi.SPX_MIXED, record=True, tuning=capi.Tuning(*tuning))
    b = run_problems(pb, precision=capi.SPX_MIXED, record=True, tuning=capi.Tuning(128, 0, 8, 0))
    assert a.stats.steps == b.stats.steps and a.stats.events == b.stats.events
    for f in ("attempts", "status", "steps", "t", "pos", "mom", "pos0", "mom0"):
        assert np.array_equal(a.records[0][f], b.records[0][f]), f


@pytest.mark.parametrize("n_distros", [0, 1])
@pytest.mark.parametrize("precision", [capi.SPX_FP64, capi.SPX_MIXED])
def test_problems_added_after_a_run_get_buffers_of_their_own(built_lib, precision, n_distros):
    """The problem buffers of a context are one allocation: problems added after a run, with bins of their own or with
    no distribution at all, are in the next run as if they had been there from the first."""
    pb = cases._parker(n=40, t_end=0.05, is_=(cases.InitialSpaceFixed(), DC().vec((0.3, 0, 0))))
    pb.plugins = [e for e in pb.plugins if n_distros or e.plugin.role != P.ROLE_DISTRIBUTION]
    out = []
    for before in (1, 3):
        sim = open_problems([pb] * before, precision=precision, record=True)
        sim.MainLoop()
        for k in range(before, 3):
            sim.ctx.add_problem(pb.n_traj, pb.seed)
        sim.ctx.run()
        out.append((sim.ctx.sync().steps, [sim.ctx.records(k, 40)["pos"] for k in range(3)]))
        sim.close()
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("ulps", [20.51, 20.49, 3.6])
@pytest.mark.parametrize("flow", [cases.FORWARD, cases.BACKWARD])
@pytest.mark.parametrize("diffusion", ["held", "general"])
def test_rounding_of_small_steps_moves_no_crossing(built_lib, diffusion, flow, ulps):
    """FP64 Parker steps of some units in the last place of the position, all rounded the same way: a path without
    diffusion moves ``round(ulps)`` units a step, and ends at the step that reaches the absorbing plane."""
    c, ulp = cases, 2.0 ** -52
    u = 1.0 if flow == c.FORWARD else -1.0
    bg = (c.BackgroundUniform(), DC().double(0.0).vec((0, 0, 0)).vec((u, 0, 0)).vec((1.0, 0, 0)).double(2.0 * ulps * ulp))
    diff = (c.DiffusionFullConstant(), DC().double(0.0).double(0.0)) if diffusion == "held" else \
           (c.DiffusionKineticEnergyRadialDistancePowerLaw(),
            DC().double(0.0).double(1.0).double(0.2).double(0.5).double(1.0).double(0.1).int(0).double(1.0).double(0.1).double(4.0))
    units_away = 200_000
    pb = c._parker(n=3, bg=bg, diff=diff, flow=flow, t_end=0.2 if flow == c.FORWARD else -0.2,
                   is_=(c.InitialSpaceFixed(), DC().vec((1.0, 0, 0))),
                   bnds=[(BoundaryPlaneAbsorb(), c.B(DC(), 1, [0]).vec((1.0 + units_away * ulp, 0, 0)).vec((1.0, 0, 0)))])
    rec = run_problems(pb, precision=capi.SPX_FP64, record=True).records[0]
    assert np.array_equal(rec["steps"], ot.run_oracle(pb).traj["steps"])
    assert np.all(np.abs(rec["steps"].astype(np.int64) - -(-units_away // round(ulps))) <= 1)


def _shape(t):
    return t.block_size, t.blocks_per_sm, t.steps_per_sync, t.schedule


@pytest.mark.parametrize("kind,precision", [("uniform", capi.SPX_FP64), ("uniform", capi.SPX_MIXED), ("dipole", capi.SPX_FP64),
                                            ("dipole", capi.SPX_MIXED), ("spiral", capi.SPX_MIXED)])
def test_autotuning_leaves_few_trajectories_their_shape(built_lib, kind, precision):
    n = 700
    if kind == "uniform":
        pb = W.diffusion_uniform(n_traj=n, t_end=0.02)
    elif kind == "dipole":
        pb = W.dipole_orbits(n_traj=n, t_end=0.01 / units.unit_time)
    else:
        pb = W.gcr_modulation(n_traj=n, energies_mev=[300.0], t_max_years=0.002)[0]
    want = run_problems(pb, precision=precision, record=True)
    sim = open_problems(pb, precision=precision, record=True)
    try:
        best = sim.ctx.autotune(4000)
        shapes = []
        for k, tuning in enumerate((None, best, want.stats.tuning)):
            st = sim.MainLoop(tuning)
            shapes.append(_shape(st.tuning))
            if k == 0:
                got = sim.ctx.records(0, n)
    finally:
        sim.close()
    assert shapes == [_shape(want.stats.tuning)] * 3
    for f in ("attempts", "status", "steps", "t", "pos", "mom"):
        assert np.array_equal(got[f], want.records[0][f]), f


@pytest.mark.parametrize("precision,n", [(capi.SPX_FP64, 152 * 128 + 1), (capi.SPX_MIXED, 152 * 128 * 3 + 1)])
def test_larger_launches_take_the_tuned_shape(built_lib, precision, n):
    """One trajectory more than the launches of few trajectories have on a GB300 (152 SMs)."""
    sim = open_problems(W.diffusion_uniform(n_traj=n, t_end=0.005), precision=precision)
    try:
        best = sim.ctx.autotune(4000)
        assert _shape(sim.MainLoop().tuning) == _shape(best) and best.blocks_per_sm > 0
    finally:
        sim.close()


@pytest.mark.parametrize("kind", ["sphere_plane", "plane_sphere", "two_spheres", "box_sphere"])
def test_two_reflections_in_one_step_match_oracle(built_lib, kind):
    """Long steps that cross two reflecting boundaries at once: each mirrors with its distance and normal at the step's
    end, where the first has not moved the point yet."""
    c = cases
    sphere = (c.BoundarySphereReflect(), c.B(DC(), -1, [-1]).vec((0, 0, 0)).double(0.4))
    plane = (BoundaryPlaneReflect(), c.B(DC(), -1, [-1]).vec((0.15, 0, 0)).vec((1.0, 0.5, 0)))
    bnds = {"sphere_plane": [sphere, plane], "plane_sphere": [plane, sphere],
            "two_spheres": [sphere, (c.BoundarySphereReflect(), c.B(DC(), -1, [-1]).vec((0.2, 0, 0)).double(0.4))],
            "box_sphere": [c.BOUNDARY_CASES["box_reflect"], sphere]}[kind]
    bg = (c.BackgroundUniform(), DC().double(0.0).vec((0, 0, 0)).vec((0, 0, 0)).vec((0, 0.3, 1.0)).double(0.2))
    pb = c._parker(n=400, bg=bg, t_end=0.2, bnds=bnds, is_=(c.InitialSpaceFixed(), DC().vec((0.05, 0, 0))))
    res = run_problems(pb, precision=capi.SPX_FP64, record=True)
    ot.assert_fp64_parity(res.records[0], ot.run_oracle(pb), ot.run_oracle(pb, nudge_libm=1), distros=res.distros[0])
