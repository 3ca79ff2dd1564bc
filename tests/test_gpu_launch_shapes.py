"""How a run is launched changes no trajectory, bit for bit. Small FP64 launches take teams of lanes in blocks of one warp,
which the tests against the oracle therefore run; larger ones have one lane a trajectory in blocks of four warps, whose
lanes are repacked as trajectories end, or the work queue. Here every problem of those tests runs in all three, with enough
trajectories for several blocks; and problems whose trajectories end one by one carry what a lane holds through the
repacking: coefficients of a uniform field, a source's memory, the state of a general Butcher table."""
import numpy as np
import pytest

import test_gpu_guiding as guiding
import test_gpu_plugins as plugins
import test_oracle_plugins as cases
import test_oracle_rk as rk_cases
from spectrum_gb300 import capi
from spectrum_gb300 import workloads as W
from spectrum_gb300.datacontainer import DataContainer as DC
from spectrum_gb300.plugins import BoundaryPlaneAbsorb
from spectrum_gb300.simulation import run_problems

pytestmark = pytest.mark.gpu

ONE_LANE, QUEUE, WIDE = capi.Tuning(128, 0, 0, 0), capi.Tuning(64, 0, 4, 1), capi.Tuning(64, 0, 8, 1)
FIELDS = ("attempts", "status", "steps", "t", "pos", "mom", "pos0", "mom0", "amp", "logwgt")


def _same_runs(pb, precision, tunings):
    a = run_problems(pb, precision=precision, record=True)
    for tuning in tunings:
        b = run_problems(pb, precision=precision, record=True, tuning=tuning)
        assert (a.stats.trajectories, a.stats.steps, a.stats.retries, a.stats.events) == \
               (b.stats.trajectories, b.stats.steps, b.stats.retries, b.stats.events)
        for f in FIELDS:
            assert a.records[0][f].tobytes() == b.records[0][f].tobytes(), f
        for (ca, _, na), (cb, _, nb) in zip(a.distros[0], b.distros[0]):
            assert na == nb and np.array_equal(ca, cb)
    return a


PROBLEMS = dict(plugins.PROBLEMS)
PROBLEMS.update({"table_" + k: v for k, v in rk_cases.RK_CASES.items()})
PROBLEMS.update({"fieldline_" + k: v for k, v in cases.FIELDLINE_CASES.items()})
PROBLEMS.update({
    "guiding_dipole": lambda: guiding.make_golden._guiding_dipole(128),
    "guidingscatt_slab": lambda: guiding.make_golden._slab_between_mirrors(guiding.TRAJ_GUIDING_SCATT, 256, d0=0.5),
    "guidingdiff_dipole": lambda: guiding.make_golden._guiding_perp(guiding.TRAJ_GUIDING_DIFF, 64, dipole=True),
    "grid": lambda: W.gcr_modulation_grid(n_traj=64, n_nodes=48, energies_mev=[300.0], t_max_years=0.02)[0],
    "blocks": lambda: W.gcr_modulation_blocks(n_traj=64, n_blocks=12, ghost_cells=0, energies_mev=[300.0], t_max_years=0.02)[0],
})
# more than 20,000 steps one after the other; others of their kind stay, and sources below
for _name in ("wnlt_constant_guiding_diff_scatt_dipole", "parker_source", "parker_source_spherical", "table_parker_source_rk29",
              "table_lorentz_dipole_rk9", "table_lorentz_dipole_rk12", "divergence_flow"):
    del PROBLEMS[_name]


@pytest.mark.parametrize("name", sorted(PROBLEMS))
def test_fp64_shapes_agree(built_lib, name):
    pb = PROBLEMS[name]()
    pb.n_traj = 300
    _same_runs(pb, capi.SPX_FP64, (ONE_LANE, QUEUE))


def _ends_one_by_one(kind, t_shock=-0.3):
    c = cases
    ball = (c.BoundarySphereAbsorb(), c.B(DC(), 1, [0]).vec((0, 0, 0)).double(0.5))
    planes = [(BoundaryPlaneAbsorb(), c.B(DC(), 1, [0]).vec((s * 0.3, 0, 0)).vec((1.0, 0, 0))) for s in (-1.0, 1.0)]
    small = (c.DiffusionFullConstant(), DC().double(0.01).double(0.02))
    if kind == "uniform":
        return c._parker(n=700, diff=(c.DiffusionFullConstant(), DC().double(0.5).double(2.0)), bnds=[ball], t_end=2.0)
    if kind == "uniform_source":
        return c._parker(n=700, traj=c.TRAJ_PARKER_SOURCE, flow=c.BACKWARD, bnds=[ball], t_end=-2.0,
                         src=(c.SourceConstant(), DC().double(0.7)))
    if kind == "shock_source":
        return c._parker(n=700, traj=c.TRAJ_PARKER_SOURCE, flow=c.BACKWARD, bg=c._shock(), diff=small, bnds=planes, t_end=t_shock,
                         src=(c.SourceMomentumInjection(), DC().double(1.0).double(2.0)),
                         im=(c.InitialMomentumShell(), DC().double(0.95)))
    if kind == "table_uniform":
        return rk_cases._with_rk(_ends_one_by_one("uniform"), 25)
    if kind == "table_shock_source":
        return rk_cases._with_rk(_ends_one_by_one("shock_source", -0.1), 29)
    pb = rk_cases._coarse_dipole(guiding.make_golden._dipole_reference_classes(400))  # Lorentz
    return rk_cases._with_rk(pb, 29)


def _repacked(steps):
    """Blocks of 128 trajectories in which 32 end more than two 64-step intervals before the last."""
    return sum(np.sort(b)[31] + 128 < b.max() for b in np.split(steps.astype(np.int64), range(128, len(steps), 128)) if len(b) == 128)


@pytest.mark.parametrize("kind", ["uniform", "uniform_source", "shock_source", "table_uniform", "table_shock_source", "table_lorentz"])
def test_repacked_lanes_keep_their_state_fp64(built_lib, kind):
    a = _same_runs(_ends_one_by_one(kind), capi.SPX_FP64, (ONE_LANE, QUEUE))
    assert _repacked(a.records[0]["steps"]) > 0


@pytest.mark.parametrize("kind", ["uniform", "uniform_source", "shock_source"])
def test_repacked_lanes_keep_their_state_fp32(built_lib, kind):
    a = _same_runs(_ends_one_by_one(kind), capi.SPX_MIXED, (WIDE,))
    assert a.stats.tuning.block_size == 128 and _repacked(a.records[0]["steps"]) > 0
