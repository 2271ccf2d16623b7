"""Full-domain sweeps where a warp owns several boxes (more boxes than resident
warps: its loop over them, resting boxes skipped, the copy back of several) and
at heights around multiples of a box's own 8 rows, against the oracle bit for
bit; and a sweep costs the same whatever the limit on their number."""

import numpy as np
import pytest
import torch

import soilb200
from oracle import relax as R
from soilb200 import _lib

pytestmark = pytest.mark.gpu

SPACING = (0.05, 0.08)
CRIT = float(np.tan(np.deg2rad(33.0)))
K = 28


def sweep(grid, iterations, tol=1e-8):
    st = _lib.RelaxStats()
    _lib.check(grid.ctx, _lib.load().sb_relax_full(
        grid.ctx, _lib.RelaxParams(*SPACING, CRIT, tol, iterations, 0), st), "relax")
    return st


def device_grid(shape, precision):
    return soilb200.DeviceGrid(shape, SPACING[1], SPACING[0], precision=precision,
                               height_exponent=K)


def heaps(ny, nx):
    """Steep heaps on flat ground: most boxes rest, those beside the heaps wake."""
    ys, xs = np.indices((ny, nx))
    h = np.zeros((ny, nx))
    for cy, cx in ((0.2, 0.15), (0.8, 0.9), (0.5, 0.5)):
        h += np.maximum(0.0, 1.0 - 0.12 * np.hypot(ys - cy * ny, xs - cx * nx))
    return h


@pytest.mark.parametrize("precision", ["fp64", "fx32"])
@pytest.mark.parametrize("shape,iterations", [
    ((1100, 1030), 11), ((1100, 1030), 12),   # 138 x 22 boxes
    ((520, 530), 70),                         # 65 x 12
    ((7, 47), 400), ((8, 48), 400), ((9, 49), 400), ((23, 95), 400), ((24, 96), 400),
    ((25, 97), 400)])
def test_sweeps_match_oracle(shape, iterations, precision):
    h = heaps(*shape)
    grid = device_grid(shape, precision)
    grid.upload("b_eff", h)
    st = sweep(grid, iterations)
    out = grid.download("b_eff")
    grid.close()
    if precision == "fp64":
        want, it, conv, *_ = R.relax_critical_slope(h, SPACING, 33.0, iterations, 1e-8)
    else:
        q = np.rint(h * 2.0 ** K).astype(np.int64)
        wq, it, conv = R.relax_critical_slope_fixed(q, SPACING, CRIT, 2.0 ** -K, iterations, 1e-8)
        want = wq * 2.0 ** -K
    assert (st.iterations, bool(st.converged)) == (it, conv)
    assert np.array_equal(out, want)


@pytest.mark.parametrize("shape", [(512, 512), (701, 701), (1024, 1024)])
def test_a_sweep_costs_the_same_under_any_limit(shape):
    """A relaxation that may run long takes the kernel of one that may not: its
    sweeps are not the slower for it (bound: a sweep's time varies by about 5 %
    between runs, the number of sweeps by 1 in 60)."""
    h = np.random.default_rng(5).random(shape)  # moves everywhere for many sweeps
    grid = device_grid(shape, "fx32")
    stream = torch.cuda.ExternalStream(grid.stream_handle())

    def time_ms(iterations):
        took = []
        for _ in range(7):
            grid.upload("b_eff", h)
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            e0.record(stream)
            assert sweep(grid, iterations).iterations == iterations
            e1.record(stream)
            e1.synchronize()
            took.append(e0.elapsed_time(e1))
        return float(np.median(took))

    time_ms(60)
    short, long = time_ms(60), time_ms(70)
    grid.close()
    assert long / 70 <= 1.25 * short / 60, (short, long)
