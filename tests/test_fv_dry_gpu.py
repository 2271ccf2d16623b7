"""The persistent substep loop skips dry blocks; the per-substep launches
(SOILB200_FV_PERSISTENT=0) visit every cell.  Both give the same fields bit for
bit: material at block, strip and domain corners, a layer that falls dry and is
wetted again (stale contents of the other buffer), chunks of one, two and eight
blocks, mostly wet and mostly dry grids."""

import numpy as np
import pytest

import soilb200
from soilb200.bulk_state import B200BulkState, B200ProductionMobileV2Solver

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def play(monkeypatch, shape, rows, persistent, layers):
    monkeypatch.setenv("SOILB200_FV_ROWS", str(rows))
    monkeypatch.setenv("SOILB200_FV_PERSISTENT", "1" if persistent else "0")
    ys, xs = np.indices(shape)
    b = 0.03 * xs + 0.2 * np.sin(ys / 9.0) * np.cos(xs / 7.0)
    state = B200BulkState(shape, 0.05, 0.05, b, mobile_headroom_m=2.0)
    solver = B200ProductionMobileV2Solver(state=state, config=soilb200.MobileV2Config(
        basal_friction_coefficient=0.2))
    out = []
    for h in layers:
        state.grid.upload("mobile", h)
        state.grid.upload("momentum_x", 0.4 * h)
        state.grid.upload("momentum_y", -0.7 * h)
        for _ in range(3):
            rec = solver.step_resident(DT)
            out += [rec.substeps, rec.volume_after_m3, rec.maximum_speed_m_s]
        out += [state.grid.download(f) for f in ("mobile", "momentum_x", "momentum_y")]
    state.close()
    return out


@pytest.mark.parametrize("rows", [5, 20, 37, 128, 200])
@pytest.mark.parametrize("shape", [(41, 29), (130, 91), (300, 64)])
def test_dry_blocks_change_nothing(monkeypatch, shape, rows):
    ys, xs = np.indices(shape)
    spots = np.zeros(shape)
    for r, c in ((0, 0), (shape[0] - 1, shape[1] - 1), (min(16, shape[0] - 1), 29 % shape[1]),
                 (shape[0] // 2, shape[1] // 2)):
        spots[r, c] = 0.3
    half = np.where(ys < shape[0] // 2, 0.2, 0.0)
    layers = [spots, np.zeros(shape), np.roll(spots, (7, 11), (0, 1)), half,
              np.full(shape, 0.15), spots]
    got = play(monkeypatch, shape, rows, True, layers)
    want = play(monkeypatch, shape, rows, False, layers)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
