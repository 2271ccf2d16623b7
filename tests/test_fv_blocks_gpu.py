"""How the substep loop starts: the ledger before a step counts the threads whose
cells are wet, and lanes without a cell (narrow grids, the end of a row) are
neither wet nor dry."""

import numpy as np
import pytest

import soilb200
from soilb200.bulk_state import B200BulkState, B200ProductionMobileV2Solver

pytestmark = pytest.mark.gpu


SHAPES = [(200, 8), (64, 16), (40, 40), (33, 64), (50, 130), (9, 300)]
# a thread of the last four sees one row (the first two give a warp several rows,
# whose majority a part of the rows does not tell)
PART = SHAPES[2:]


@pytest.mark.parametrize("shape,wet_rows,mode",
                         [(s, 0.0, 0) for s in SHAPES] + [(s, 1.0, 2) for s in SHAPES]
                         + [(s, 0.3, 0) for s in PART] + [(s, 0.7, 1) for s in PART])
def test_first_substep_mode(shape, wet_rows, mode):
    ys, xs = np.indices(shape)
    b = 0.03 * xs + 0.2 * np.sin(ys / 9.0)
    state = B200BulkState(shape, 0.05, 0.05, b, mobile_headroom_m=2.0)
    solver = B200ProductionMobileV2Solver(state=state, config=soilb200.MobileV2Config(
        basal_friction_coefficient=0.2))
    chunk, rows, cols, _ = state.grid.fv_blocks()
    assert 1 <= rows <= chunk and cols == 30
    state.grid.upload("mobile", np.where(ys < wet_rows * shape[0], 0.2, 0.0))
    solver.step_resident(1.0 / 60.0)
    assert state.grid.fv_blocks()[3] == mode
    state.close()


def test_no_loop_no_blocks():
    grid = soilb200.DeviceGrid((40, 40), 0.05, 0.05, precision="fp64")
    assert grid.fv_blocks() == (0, 0, 0, 0)
    grid.close()
