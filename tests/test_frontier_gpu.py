"""The one-launch compact frontier where its index ranges end: tile sizes of one
cell, odd and larger than the grid, ragged last tiles, runs that follow one
another on the same grid, and the round limit.  FP64, bit-identical to the
oracle's schedule with equal round counts."""

import numpy as np
import pytest

import soilb200
from oracle import relax as R

pytestmark = pytest.mark.gpu

CRIT = float(np.tan(np.deg2rad(33.0)))


def event(shape, seed):
    rng = np.random.default_rng([seed, *shape])
    h = 0.5 + 0.002 * rng.random(shape)
    seeds = np.zeros(shape, dtype=bool)
    for _ in range(4):
        r, c = rng.integers(0, shape[0]), rng.integers(0, shape[1])
        sl = (slice(max(r - 1, 0), r + 2), slice(max(c - 1, 0), c + 2))
        h[sl] += rng.uniform(0.2, 0.4)
        seeds[sl] = True
    return h, seeds


@pytest.mark.parametrize("tile", [1, 2, 5, 16, 33, 64])
@pytest.mark.parametrize("shape", [(2, 2), (17, 40), (65, 31)])
def test_frontier_matches_oracle(shape, tile):
    w = R.vertex_weights(shape, 0.05, 0.05)
    grid = soilb200.DeviceGrid(shape, 0.05, 0.05, precision="fp64", tile_size=tile)
    front = soilb200.FrontierRelaxation(grid, weighted=True)
    for seed in (1, 2):
        h, seeds = event(shape, seed)
        want, _, rounds, _ = R.frontier_relax(h, seeds, R.seed_tiles(seeds, tile), tile=tile,
                                              spacing=(0.05, 0.05), crit_tan=CRIT,
                                              tolerance=1e-8, weights=w)
        grid.upload("b_eff", h)
        front.seed_mask(seeds)
        st = front.run(CRIT, 1e-8)
        assert (st.rounds, st.converged, st.active_tiles_last_round) == (rounds, True, 0)
        assert np.array_equal(grid.download("b_eff"), want)
        assert not grid.download("frontier_reached").any()
        assert front.active_tiles().size == 0
    grid.close()


def test_round_limit_then_a_fresh_run():
    shape, tile = (40, 50), 8
    h, seeds = event(shape, 3)
    grid = soilb200.DeviceGrid(shape, 0.05, 0.05, precision="fp64", tile_size=tile)
    front = soilb200.FrontierRelaxation(grid, weighted=True)
    grid.upload("b_eff", h)
    front.seed_mask(seeds)
    with pytest.raises(soilb200.NumericalNonconvergenceError):
        front.run(CRIT, 1e-8, 2)
    grid.upload("b_eff", h)
    grid.upload("frontier_reached", np.zeros(shape, np.int32))
    front.seed_mask(seeds)
    want, _, rounds, _ = R.frontier_relax(h, seeds, R.seed_tiles(seeds, tile), tile=tile,
                                          spacing=(0.05, 0.05), crit_tan=CRIT, tolerance=1e-8,
                                          weights=R.vertex_weights(shape, 0.05, 0.05))
    assert front.run(CRIT, 1e-8).rounds == rounds
    assert np.array_equal(grid.download("b_eff"), want)
    grid.close()
