"""Densities whose weight terms leave float32's normal range: the shortcut of
calm cells must not apply (its margins are rounding's there), and severity and
labels are the oracle's float32 operations bit for bit."""

import numpy as np
import pytest

import soilb200
from oracle import fixed_point as fx
from oracle import labels as L

pytestmark = pytest.mark.gpu

DX, K = 0.05, 24


@pytest.mark.filterwarnings("ignore::RuntimeWarning")  # the oracle overflows as the kernel does
@pytest.mark.parametrize("start,stop", [(38.0, 30.0), (30.0, 38.0)])
@pytest.mark.parametrize("density", [1e-39, 1e-37, 1e-36, 1e-18, 1370.0, 1e18, 1e36])
def test_yield_at_the_ends_of_float32(density, start, stop):
    ny, nx = 70, 66
    rng = np.random.default_rng(11)
    b = np.cumsum(0.8 * DX * rng.random((ny, nx)), axis=1)
    z = b - np.exp(rng.uniform(np.log(2.0 ** -K), 0.0, (ny, nx)))
    zero = np.zeros((ny, nx))
    grid = soilb200.DeviceGrid((ny, nx), DX, DX, precision="fx32", height_exponent=K)
    grid.upload("b_eff", b)
    grid.upload("z_base", z)
    bridge = soilb200.B200LargeAvalancheBridge(
        grid, soilb200.MaterialScenario("m", density, 29.8, 0.0, 0.5, start, stop, 0.35))
    bridge.label(release_settled_latches=False)
    want = L.yield_init(fx.quantize(b, 0.0, K), fx.quantize(z, 0.0, K), fx.quantize(zero, 0.0, K),
                        None, None, dx=DX, dy=DX, tan_start=np.tan(np.deg2rad(start)),
                        tan_stop=np.tan(np.deg2rad(stop)), density=density, gravity=9.81,
                        cohesion=0.0, mobilization_depth=0.08, dry=1e-8, fixed_point=True,
                        quantum=2.0 ** -K)
    assert np.array_equal(grid.download("severity").astype(np.float32), want["severity"])
    assert np.array_equal(bridge.labels(), L.canonical_labels(want["unstable"], 8))
    grid.close()
