"""A proposal is queued on the grid's stream and returns at once.  Dropping the
object that queued it frees the proposal's buffers to other streams, so the drop
waits for it."""

import numpy as np
import pytest
import torch

import soilb200
from soilb200 import learned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused", [True, False])
def test_dropping_the_object_waits_for_its_proposals(fused):
    shape = (1500, 1500)  # a round takes about 150 us, the drop some microseconds
    grid = soilb200.DeviceGrid(shape, 0.05, 0.05, precision="fx32", height_exponent=28)
    grid.upload("b_eff", np.random.default_rng(3).random(shape))
    lr = learned.LearnedRelaxation(grid, learned.ReposeNet(seed=1), 35.0, fused=fused)
    stream = torch.cuda.ExternalStream(grid.stream_handle())
    lr.propose(2)
    grid.synchronize()
    lr.propose(40)
    del lr
    assert stream.query()
    grid.close()


def test_the_grid_may_close_first():
    grid = soilb200.DeviceGrid((70, 90), 0.05, 0.05, precision="fx32", height_exponent=28)
    lr = learned.LearnedRelaxation(grid, learned.ReposeNet(seed=1), 35.0)
    lr.propose(3)
    grid.close()
    del lr
    torch.cuda.synchronize()


def test_weights_are_those_of_the_making():
    """Weights written on the caller's stream just before are the ones taken, and
    a change after the making is not seen."""
    rng = np.random.default_rng(2)
    b = 0.3 * rng.random((64, 64))
    outs = []
    for late in (False, True):
        net = learned.ReposeNet(seed=1)
        with torch.cuda.stream(torch.cuda.Stream()):
            for w in net.weights:
                w.mul_(1.5)
            grid = soilb200.DeviceGrid(b.shape, 0.05, 0.05, precision="fx32", height_exponent=28)
            grid.upload("b_eff", b)
            lr = learned.LearnedRelaxation(grid, net, 35.0)
            if late:
                for w in net.weights:
                    w.zero_()
        lr.propose(2)
        outs.append(grid.download("b_eff"))
        grid.close()
    assert not np.array_equal(outs[0], b)
    assert np.array_equal(outs[0], outs[1])
