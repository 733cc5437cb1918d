"""A velocity that is NaN in every cell, as one Poisson solve leaves it after
any NaN: the step reports CUP2D_ENAN, and the time and the next dt it leaves
are numbers -- findMaxU takes no NaN, so the dt is the one its full-grid scan
gives (the viscous and body limits)."""
import numpy as np
import pytest

from cubismup_2d_b200 import Cup2DError, Simulation, abi

pytestmark = pytest.mark.gpu

ARGS = ("-bpdx 4 -bpdy 2 -extent 1 -CFL 0.1 -nu 1e-3 -lambda 1e4 -poissonType freespace "
        "-muteAll 1 -shapes 'disk radius=0.1 xpos=0.3 ypos=0.25 bForced=1 bFixed=1 xvel=0.2'")


def _all_nan():
    s = Simulation(ARGS)
    s.init()
    for _ in range(2):
        s.advance(s.calcMaxTimestep())
    dt = s.calcMaxTimestep()
    nan = np.full((s.ctx.ny, s.ctx.nx), np.nan)
    s.ctx.set("u", nan)
    s.ctx.set("v", nan)
    return s, dt


def _scanned_dt(s):
    s.ctx.set("u", s.ctx.get("u"))          # the carried dt no longer holds: a scan of the grid
    return s.calcMaxTimestep()


def _expect_nan_status(s):
    with pytest.raises(Cup2DError) as e:
        s.ctx.sync()
    assert e.value.code == abi.ENAN


def test_operator_step_leaves_a_finite_dt():
    s, dt = _all_nan()
    for op in s.pipeline:
        op(dt)
    s.ctx.end_step()
    carried = s.calcMaxTimestep()           # formed by the step's own kernels
    assert np.isfinite(carried) and carried == _scanned_dt(s)
    assert np.isfinite(s.ctx.scalars()["time"])
    _expect_nan_status(s)


def test_graph_steps_leave_a_finite_time():
    s, _ = _all_nan()
    s.ctx.advance(2)                        # the second step takes the dt the first one formed
    sc = s.ctx.scalars()
    assert np.isfinite(sc["time"]) and np.isfinite(sc["dt"])
    _expect_nan_status(s)
