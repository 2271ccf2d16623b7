"""Sweeps of one call each against the same number in one call: both height
buffers, the copy back after an odd number and the barrier's words from call to
call."""

import numpy as np
import pytest

import soilb200
from soilb200 import _lib

pytestmark = pytest.mark.gpu

SPACING = (0.05, 0.08)
CRIT = float(np.tan(np.deg2rad(33.0)))


@pytest.mark.parametrize("precision", ["fp64", "fx32"])
@pytest.mark.parametrize("count", [1, 2, 3, 8])
@pytest.mark.parametrize("shape", [(3, 5), (130, 200), (300, 61)])
def test_single_sweeps_equal_one_call(shape, count, precision):
    lib = _lib.load()
    h = np.random.default_rng(list(shape)).random(shape)
    h[shape[0] // 2:] = 0.5  # the lower half rests at first
    out = []
    for parts in ([count], [1] * count, [count - count // 2, count // 2]):
        grid = soilb200.DeviceGrid(shape, SPACING[1], SPACING[0], precision=precision,
                                   height_exponent=28)
        grid.upload("b_eff", h)
        for n in parts:
            if n:
                assert lib.sb_relax_sweeps(
                    grid.ctx, _lib.RelaxParams(*SPACING, CRIT, 0.0, n, 0)) == _lib.SB_OK
        out.append(grid.download("b_eff"))
        grid.close()
    assert not np.array_equal(out[0], h)
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
