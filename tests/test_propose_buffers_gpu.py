"""A proposal is queued on the grid's stream and may still run when the object
that queued it is gone: its buffers belong to that stream, so that the allocator
does not give them to work of another stream meanwhile."""

import numpy as np
import pytest
import torch

import soilb200
from soilb200 import learned

pytestmark = pytest.mark.gpu


def _stream_of(tensor) -> int:
    p = tensor.data_ptr()
    for seg in torch.cuda.memory_snapshot():
        if seg["address"] <= p < seg["address"] + seg["total_size"]:
            return int(seg["stream"])
    raise AssertionError("not the allocator's memory")


@pytest.mark.parametrize("fused", [True, False])
def test_buffers_belong_to_the_grids_stream(fused):
    grid = soilb200.DeviceGrid((70, 90), 0.05, 0.05, precision="fx32", height_exponent=28)
    lr = learned.LearnedRelaxation(grid, learned.ReposeNet(seed=1), 35.0, fused=fused)
    held = [v for k, v in vars(lr).items() if isinstance(v, torch.Tensor)] + list(lr._packed)
    assert len(held) >= 6
    assert {_stream_of(t) for t in held} == {grid.stream_handle()}
    grid.close()


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
