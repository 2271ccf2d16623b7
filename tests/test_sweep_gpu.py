"""The sweep kernel where its boxes end: a warp's box is 32 x 64 cells of which
16 x 48 are its own, tiles at rest are skipped, and heights beyond +-2^30 quanta
take the wide arithmetic.  Bit-identical to the oracle, iteration counts equal."""

import numpy as np
import pytest

import soilb200
from oracle import relax as R
from soilb200 import _lib

pytestmark = pytest.mark.gpu

SPACING = (0.05, 0.08)
CRIT = float(np.tan(np.deg2rad(33.0)))
K = 28


def run(field, precision, iterations, tol=1e-8):
    grid = soilb200.DeviceGrid(field.shape, SPACING[1], SPACING[0], precision=precision,
                               height_exponent=K)
    try:
        grid.upload("b_eff", field)
        p = _lib.RelaxParams(*SPACING, CRIT, tol, iterations, 0)
        st = _lib.RelaxStats()
        _lib.check(grid.ctx, _lib.load().sb_relax_full(grid.ctx, p, st), "relax")
        return grid.download("b_eff"), st
    finally:
        grid.close()


def surface(ny, nx, rough):
    """Two steep heaps far apart on flat ground (tiles between them rest, then wake)."""
    rng = np.random.default_rng([ny, nx])
    ys, xs = np.indices((ny, nx))
    h = 0.3 * rough * rng.random((ny, nx))
    for cy, cx in ((0.2 * ny, 0.15 * nx), (0.8 * ny, 0.9 * nx)):
        h += np.maximum(0.0, 1.0 - 0.12 * np.hypot(ys - cy, xs - cx))
    return h


@pytest.mark.parametrize("precision", ["fp64", "fx32"])
@pytest.mark.parametrize("iterations", [1, 2, 7, 5000])
@pytest.mark.parametrize("shape", [(2, 2), (2, 131), (97, 3), (16, 48), (17, 49), (15, 47),
                                   (33, 64), (40, 113), (129, 200)])
def test_sweeps_match_oracle(shape, iterations, precision):
    h = surface(*shape, rough=shape[0] % 2)
    out, st = run(h, precision, iterations)
    if precision == "fp64":
        want, it, conv, *_ = R.relax_critical_slope(h, SPACING, 33.0, iterations, 1e-8)
    else:
        q = np.rint(h * 2.0 ** K).astype(np.int64)
        wq, it, conv = R.relax_critical_slope_fixed(q, SPACING, CRIT, 2.0 ** -K, iterations, 1e-8)
        want = wq * 2.0 ** -K
    assert st.iterations == it and bool(st.converged) == conv
    assert np.array_equal(out, want)


@pytest.mark.parametrize("tol", [0.0, 2.0 ** -K, 1e-3])
def test_tolerances_match_oracle(tol):
    h = surface(60, 70, 1)
    q = np.rint(h * 2.0 ** K).astype(np.int64)
    wq, it, conv = R.relax_critical_slope_fixed(q, SPACING, CRIT, 2.0 ** -K, 300, tol)
    out, st = run(h, "fx32", 300, tol)
    assert (st.iterations, bool(st.converged)) == (it, conv)
    assert np.array_equal(out, wq * 2.0 ** -K)
    want, it, conv, *_ = R.relax_critical_slope(h, SPACING, 33.0, 300, tol)
    out, st = run(h, "fp64", 300, tol)
    assert (st.iterations, bool(st.converged)) == (it, conv)
    assert np.array_equal(out, want)


def test_heights_over_the_whole_int32_range():
    rng = np.random.default_rng(3)
    q = rng.integers(-2 ** 31 + 1, 2 ** 31 - 1, (70, 100))
    q[:, :40] = rng.integers(-2 ** 28, 2 ** 28, (70, 40))  # narrow tiles beside wide ones
    wq, it, conv = R.relax_critical_slope_fixed(q, SPACING, CRIT, 2.0 ** -K, 40, 1e-8)
    out, st = run(q * 2.0 ** -K, "fx32", 40)
    assert (st.iterations, bool(st.converged)) == (it, conv)
    assert np.array_equal(out, wq * 2.0 ** -K)
