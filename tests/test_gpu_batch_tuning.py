"""Fixed steps on the stage GEMM run by a rule on the sizes; no call times the
alternatives on its way, however many steps it has (that cost 58 to 81 steps for
picks no faster than the rule's).  mpc_batch_autotune does on request.
"""
import numpy as np
import pytest

import mpc_tdse
from mpc_tdse.systems import random_system

pytestmark = pytest.mark.gpu


def test_fixed_steps_do_not_tune_unasked():
    s = random_system([60, 70, 50], gauge="l", seed=3, e_max=8.0, d_scale=0.3)
    Io, w = mpc_tdse.to_au(2e14, 4.0)
    p = mpc_tdse.pulse_setup("sine", "l", Io, w, 0.0, 2, mpc_tdse.period(w, 2))
    X = np.zeros((12, s.ntot), complex)
    X[:, 0] = 1.0
    with mpc_tdse.Context.from_system(s) as ctx:
        ctx.set_path("streaming")
        assert ctx.batch_fixed_plan() == []
        ctx.batch_advance([p] * 12, 0.0, 0.05, [3] * 12, X)
        plan = ctx.batch_fixed_plan()
        assert [r[0] for r in plan] == [1, 2, 4, 8, 16]
        Y = ctx.batch_advance([p] * 12, 0.0, 0.05, [600] * 12, X)
        assert ctx.batch_fixed_plan() == plan and all(r[4] == 0 for r in plan)
        ctx.batch_autotune(12)
        timed = ctx.batch_fixed_plan()
        assert [r[0] for r in timed] == [1, 2, 4, 8, 16] and all(r[4] > 0 for r in timed)
        assert np.array_equal(ctx.batch_advance([p] * 12, 0.0, 0.05, [600] * 12, X), Y)


def test_autotune_reports_the_widths_it_was_asked_for():
    """A long adaptive call has tuned its own width (40 pulses: the bucket of 64)
    and none below; the table for 4 pulses has the rows 1, 2, 4."""
    s = random_system([60, 70, 50], gauge="l", seed=3, e_max=8.0, d_scale=0.3)
    Io, w = mpc_tdse.to_au(2e14, 4.0)
    p = mpc_tdse.pulse_setup("sine", "l", Io, w, 0.0, 2, mpc_tdse.period(w, 2))
    X = np.zeros((40, s.ntot), complex)
    X[:, 0] = 1.0
    with mpc_tdse.Context.from_system(s) as ctx:
        ctx.set_path("streaming")
        ctx.batch_propagate([p] * 40, 0.0, [21.0] * 40, X, dt_max=0.1)
        rows = ctx.batch_autotune(4)
    assert [r[0] for r in rows] == [1, 2, 4]
    assert all(r[1] in (16, 32, 64) and r[2] in (3, 6) and r[4] > 0 for r in rows)
