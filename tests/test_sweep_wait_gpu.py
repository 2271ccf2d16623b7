"""A sweep whose CTAs give up waiting for one another: the call, or for queued
sweeps the next one that reports, fails with the wait's status, and the one after
that is a relaxation like any other.  No poll at all is allowed here, so that the
first CTA at the barrier leaves at once."""

import numpy as np
import pytest

import soilb200
from oracle import relax as R
from soilb200 import _lib

pytestmark = pytest.mark.gpu

DX = 0.05
CRIT = float(np.tan(np.deg2rad(33.0)))
K = 28
SHAPE = (200, 210)  # 25 x 5 boxes, 32 CTAs


def _grid():
    return soilb200.DeviceGrid(SHAPE, DX, DX, precision="fx32", height_exponent=K)


def _params(iterations):
    return _lib.RelaxParams(DX, DX, CRIT, 1e-8, iterations, 0)


def _full(grid, iterations):
    st = _lib.RelaxStats()
    _lib.check(grid.ctx, _lib.load().sb_relax_full(grid.ctx, _params(iterations), st), "relax")
    return st


@pytest.mark.parametrize("queued", [0, 1, 3])
def test_a_wait_that_gave_up_is_reported_once(queued):
    lib = _lib.load()
    h = np.random.default_rng(8).random(SHAPE)
    grid = _grid()
    grid.upload("b_eff", h)
    assert lib.sb_relax_wait_polls(grid.ctx, 0) == _lib.SB_OK
    for _ in range(queued):  # return at once: the status stays on the device
        assert lib.sb_relax_sweeps(grid.ctx, _params(4)) == _lib.SB_OK
    if queued:
        lib.sb_relax_wait_polls(grid.ctx, -1)
        # sweeps that run through in between do not wipe it out
        assert lib.sb_relax_sweeps(grid.ctx, _params(2)) == _lib.SB_OK
    with pytest.raises(RuntimeError, match="wait gave up"):
        _full(grid, 6)
    lib.sb_relax_wait_polls(grid.ctx, -1)
    grid.upload("b_eff", h)
    st = _full(grid, 6)
    q = np.rint(h * 2.0 ** K).astype(np.int64)
    want, it, conv = R.relax_critical_slope_fixed(q, (DX, DX), CRIT, 2.0 ** -K, 6, 1e-8)
    assert (st.iterations, bool(st.converged), st.status) == (it, conv, 0)
    assert np.array_equal(grid.download("b_eff"), want * 2.0 ** -K)
    grid.close()
