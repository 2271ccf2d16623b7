"""The fixed-point ledger and yield kernels where their shortcuts end.

* Ledger: a warp takes 128 columns as 16-byte words and border cells' weights go
  a separate way: widths and heights at their edges, against NumPy sums of the
  stored fields (integer sums equal; float64 sums of n terms to 2 n 2^-53 of the
  sum of magnitudes).
* Static short-circuit: a float32 gradient settles a cell below the start slope
  by 1e-4, the others are taken in FP64: one quantum decides, wherever it stands.
* Yield: cells below both tangents by 1e-5 skip the margins: the same bits as
  the margins' oracle on slopes around that line.
"""

import numpy as np
import pytest

import soilb200
from oracle import fixed_point as fx
from oracle import labels as L
from oracle.relax import vertex_weights6
from soilb200 import _lib
from soilb200.mobile_v2 import mobile_params

pytestmark = pytest.mark.gpu

DX, DY, K = 0.05, 0.04, 24
Q = 2.0 ** -K


def _grid(shape, b, z, h, qx, qy):
    grid = soilb200.DeviceGrid(shape, DX, DY, precision="fx32", height_exponent=K)
    for name, f in (("b_eff", b), ("z_base", z), ("mobile", h), ("momentum_x", qx),
                    ("momentum_y", qy)):
        grid.upload(name, f)
    return grid


@pytest.mark.parametrize("wet", [0.0, 0.15, 1.0])
@pytest.mark.parametrize("shape", [(2, 2), (3, 5), (5, 127), (6, 128), (7, 129), (40, 132),
                                   (33, 389), (700, 3)])
def test_ledger_sums(shape, wet):
    rng = np.random.default_rng(shape[0] * 1000 + shape[1])
    on = rng.random(shape) < wet
    b, z = rng.normal(size=shape), rng.normal(size=shape)
    h = np.where(on, 0.3 * rng.random(shape), 0.0)
    qx = np.where(on, rng.normal(size=shape), -0.0)  # a momentum of -0 is none
    qy = np.where(on & (rng.random(shape) < 0.5), rng.normal(size=shape), 0.0)
    grid = _grid(shape, b, z, h, qx, qy)
    params = mobile_params(soilb200.MobileV2Config(dx_m=DX, dy_m=DY), density_kg_m3=1.0)
    got = _lib.MobileLedger()
    _lib.check(grid.ctx, _lib.load().sb_mobile_ledger_of(grid.ctx, params, got), "ledger")
    bq, zq, hq = (grid.download(n) for n in ("b_eff", "z_base", "mobile"))
    grid.close()
    w6, f, rho = vertex_weights6(shape), DX * DY / 6.0, params.density_kg_m3
    hi = np.rint(hq / Q).astype(np.int64)
    rest = np.maximum(np.rint((bq - zq) / Q).astype(np.int64), 0)
    assert got.mass_quanta == hi.sum() and got.volume_w_quanta == (hi * w6).sum()
    assert got.resting_w_quanta == (rest * w6).sum()
    assert min(got.min_h_m, 0.0) == min(hq.min(), 0.0)  # as callers read it
    x, y = qx.astype(np.float32).astype(np.float64), qy.astype(np.float32).astype(np.float64)
    moving = hq > 1e-8
    e = np.where(moving, (x * x + y * y) / np.where(moving, hq, 1.0), 0.0)
    g, kg = params.gravity_m_s2, params.earth_pressure_coefficient * params.gravity_m_s2
    for value, terms in (
            (got.momentum_m4_s[0], x * DX * DY), (got.momentum_m4_s[1], y * DX * DY),
            (got.kinetic, 0.5 * e * DX * DY), (got.gravitational, g * hq * bq * DX * DY),
            (got.internal, 0.5 * kg * hq * hq * DX * DY),
            (got.momentum_w[0], rho * f * x * w6), (got.momentum_w[1], rho * f * y * w6),
            (got.kinetic_w_j, 0.5 * rho * f * e * w6), (got.potential_w_j, rho * g * f * hq * bq * w6),
            (got.pressure_w_j, 0.5 * rho * kg * f * hq * hq * w6)):
        # 8: the roundings of one term; the border share is taken off 6 times a sum
        bound = 2.0 * (terms.size + 8) * 2.0 ** -53 * 6.0 * np.abs(terms).sum()
        assert abs(value - terms.sum()) <= bound
    speed = np.sqrt((e / np.where(moving, hq, 1.0)).max())
    assert got.max_speed_m_s == pytest.approx(speed, rel=1e-15, abs=0.0)


@pytest.mark.parametrize("at", [(0, 0), (0, 64), (6, 130), (3, 0), (3, 3), (3, 4), (3, 127),
                                (3, 128), (4, 129), (6, 63)])
def test_one_quantum_decides_the_static_short_circuit(at):
    shape = (7, 131)
    params = soilb200.MobileV2Config(dx_m=DX, dy_m=DY)
    limit = np.tan(np.deg2rad(params.start_angle_deg)) + 1.0e-14

    def steepest(q):
        s = np.zeros(shape)
        s[at] = q * Q
        gy, gx = np.gradient(s, DY, DX)
        return np.hypot(gx, gy).max()

    top = int(limit / steepest(1))
    while steepest(top + 1) <= limit:
        top += 1
    while steepest(top) > limit:
        top -= 1
    zero = np.zeros(shape)
    for quanta, static in ((top, 1), (top + 1, 0), (4 * top, 0)):
        b = zero.copy()
        b[at] = quanta * Q
        grid = _grid(shape, b, zero, zero, zero, zero)
        stats = _lib.MobileStats()
        _lib.check(grid.ctx, _lib.load().sb_mobile_step(grid.ctx, 1.0 / 60.0, mobile_params(params),
                                                        stats), "step")
        grid.close()
        assert stats.static_skip == static


@pytest.mark.parametrize("start,stop,cohesion", [(38.0, 30.0, 0.0), (38.0, 30.0, 60.0),
                                                 (30.0, 38.0, 0.0), (33.0, 33.0, 0.0)])
def test_yield_around_its_calm_line(start, stop, cohesion):
    ny, nx = 66, 130
    ts, tp = np.tan(np.deg2rad(start)), np.tan(np.deg2rad(stop))
    ys, xs = np.indices((ny, nx))
    # slopes from 3e-5 below to 3e-5 above each tangent, one per row pair
    rel = np.linspace(-3e-5, 3e-5, ny)[:, None]
    b = np.where(xs < nx // 2, ts, tp) * (1.0 + rel) * DX * xs
    z = b - np.where(ys % 3 == 0, 0.0, 0.1)
    zero = np.zeros((ny, nx))
    grid = _grid((ny, nx), b, z, zero, zero, zero)
    bridge = soilb200.B200LargeAvalancheBridge(
        grid, soilb200.MaterialScenario("m", 1370.0, 29.8, cohesion, 0.5, start, stop, 0.35))
    bridge.label(release_settled_latches=False)
    bq, zq = fx.quantize(b, 0.0, K), fx.quantize(z, 0.0, K)
    want = L.yield_init(bq, zq, fx.quantize(zero, 0.0, K), None, None, dx=DX, dy=DY, tan_start=ts,
                        tan_stop=tp, density=1370.0, gravity=9.81, cohesion=cohesion,
                        mobilization_depth=0.08, dry=1e-8, fixed_point=True, quantum=Q)
    assert np.array_equal(bridge.labels(), L.canonical_labels(want["unstable"], 8))
    assert np.array_equal(grid.download("severity").astype(np.float32), want["severity"])
    grid.close()


@pytest.mark.parametrize("release", [False, True])
@pytest.mark.parametrize("shape", [(2, 2), (3, 2), (33, 31), (31, 34), (64, 36), (40, 67)])
def test_yield_quads_at_tile_and_row_edges(shape, release):
    """Four cells per thread: widths that are and are not whole quads and tiles,
    and a surface whose differences leave 32 bits (heights of +-2^31 quanta)."""
    rng = np.random.default_rng(shape[0] * 100 + shape[1])
    for scale in (0.05, 100.0):
        b = scale * rng.uniform(-1.0, 1.0, shape)
        z = b - 0.2 * rng.random(shape)
        h = np.where(rng.random(shape) < 0.3, 0.1 * rng.random(shape), 0.0)
        zero = np.zeros(shape)
        grid = _grid(shape, b, z, h, zero, zero)
        bridge = soilb200.B200LargeAvalancheBridge(
            grid, soilb200.MaterialScenario("m", 1370.0, 29.8, 0.0, 0.5, 38.0, 30.0, 0.35))
        bridge.label(release_settled_latches=release)
        want = L.yield_init(fx.quantize(b, 0.0, K), fx.quantize(z, 0.0, K), fx.quantize(h, 0.0, K),
                            None, None, dx=DX, dy=DY, tan_start=np.tan(np.deg2rad(38.0)),
                            tan_stop=np.tan(np.deg2rad(30.0)), density=1370.0, gravity=9.81,
                            cohesion=0.0, mobilization_depth=0.08, dry=1e-8, fixed_point=True,
                            quantum=Q)
        assert np.array_equal(bridge.labels(), L.canonical_labels(want["unstable"], 8))
        for name in ("slope", "severity"):
            assert np.array_equal(grid.download(name).astype(np.float32), want[name])
        grid.close()
