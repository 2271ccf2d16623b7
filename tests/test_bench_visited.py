"""The bench's count of the cells that the substep loop visits, against a walk
over the cells."""

import numpy as np
import pytest

import bench


@pytest.mark.parametrize("blocks", [(5, 5, 30), (37, 16, 30), (121, 16, 30), (200, 25, 30),
                                    (7, 3, 4)])
@pytest.mark.parametrize("shape", [(1, 1), (5, 30), (61, 47), (130, 91)])
def test_visited_cells_are_those_beside_material(shape, blocks):
    chunk, height, width = blocks
    rng = np.random.default_rng(sum(shape) + chunk)
    for wet in (0.0, 0.001, 0.01, 1.0):
        h = np.where(rng.random(shape) < wet, 0.1, 0.0)
        per = -(-chunk // height)
        row = [(r // chunk) * per + r % chunk // height for r in range(shape[0])]
        block = {(r, c): (row[r], c // width) for r in range(shape[0]) for c in range(shape[1])}
        full = {block[r, c] for r, c in zip(*np.nonzero(h))}
        near = {(i + di, j + dj) for i, j in full for di in (-1, 0, 1) for dj in (-1, 0, 1)}
        assert bench.visited_cells(h, blocks) == sum(b in near for b in block.values())


def test_one_wet_cell_of_the_default_workload():
    """701^2 has chunks of one block of 5 rows: 3 blocks by 3, not 3 x 16 rows."""
    h = np.zeros((701, 701))
    h[352, 341] = 0.2
    assert bench.visited_cells(h, (5, 5, 30, 0)) == 15 * 90
    assert bench.visited_cells(h, (0, 0, 0, 0)) == h.size
