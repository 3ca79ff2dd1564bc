"""The device buffers of a context while its problems change: they hold as many problems as the last run had, and calls
in between touch no more than that."""
import numpy as np
import pytest

from spectrum_gb300 import capi
from spectrum_gb300.simulation import open_problems
from test_gpu_dump import CASES

pytestmark = pytest.mark.gpu


def _state(sim, n):
    return [(sim.ctx.distribution(k, 0), sim.ctx.distribution_records(k, 0)[2]) for k in range(n)]


@pytest.mark.parametrize("added", [1, 40])
def test_reset_between_added_problems_and_the_next_run(built_lib, added):
    """spx_reset_distributions after problems were added clears what the last run's problems have; the next run is that
    of a context that had all problems from the first, with its run index moved on by one."""
    pb = CASES["focused_fwd_slab_records"]
    a, b = open_problems(pb, capi.SPX_FP64), open_problems([pb] * (1 + added), capi.SPX_FP64)
    try:
        a.MainLoop()
        assert _state(a, 1)[0][0][2] == 12
        for _ in range(added):
            a.ctx.add_problem(pb.n_traj, pb.seed)
        a.ctx.reset_distributions()
        assert all(n == 0 and not c.any() and not s.any() for (c, s, n), _ in _state(a, 1 + added))
        a.ctx.run()
        b.ctx.set_option(capi.SPX_OPT_RUN_INDEX, 1)
        b.ctx.run()
        assert a.ctx.sync().steps == b.ctx.sync().steps
        for (da, ra), (db, rb) in zip(_state(a, 1 + added), _state(b, 1 + added)):
            assert ra == rb and da[2] == db[2] and np.array_equal(da[0], db[0])
    finally:
        a.close()
        b.close()


def test_more_problems_at_a_smaller_record_capacity(built_lib):
    """Forty problems that keep a tenth of the records of four take as many slots, and ten times the counters."""
    pb = CASES["focused_fwd_slab_records"]
    a, b = open_problems([pb] * 4, capi.SPX_FP64), open_problems([pb] * 40, capi.SPX_FP64)
    try:
        a.ctx.set_option(capi.SPX_OPT_RECORD_CAPACITY, 100)
        a.MainLoop()
        for _ in range(36):
            a.ctx.add_problem(pb.n_traj, pb.seed)
        b.ctx.set_option(capi.SPX_OPT_RUN_INDEX, 1)
        for sim in (a, b):
            sim.ctx.set_option(capi.SPX_OPT_RECORD_CAPACITY, 10)
            sim.ctx.run()
            sim.ctx.sync()
        for (da, ra), (db, rb) in zip(_state(a, 40), _state(b, 40)):
            assert ra == rb == da[2] == db[2] and np.array_equal(da[0], db[0])
    finally:
        a.close()
        b.close()
