"""sb_learned_propose (one call, kernels overlapping their predecessors) against
the layer-by-layer round (fused=False): the same heights bit for bit, at strip
edges (122 pixels), odd sizes and heights where the transfer limit binds."""

import numpy as np
import pytest

import soilb200
from soilb200 import learned
from soilb200.train_repose import DEFAULT_WEIGHTS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 0.37, 1e6])
@pytest.mark.parametrize("shape", [(2, 2), (5, 121), (31, 122), (9, 123), (64, 245), (150, 67)])
def test_fused_round_equals_layer_launches(shape, scale):
    rng = np.random.default_rng(list(shape))
    ys, xs = np.indices(shape)
    b = np.maximum(0.0, 1.5 - 0.08 * np.hypot(ys - shape[0] / 2, xs - shape[1] / 3))
    b += 0.2 * rng.random(shape)
    net = learned.ReposeNet.load(DEFAULT_WEIGHTS)
    k, datum = soilb200.choose_quantization(b)
    out = []
    for fused in (True, False):
        grid = soilb200.DeviceGrid(shape, 0.05, 0.05, precision="fx32", height_exponent=k,
                                   datum_m=datum)
        grid.upload("b_eff", b)
        before = grid.download("b_eff")
        lr = learned.LearnedRelaxation(grid, net, 35.0, fused=fused)
        lr.propose(3, scale)
        out.append(grid.download("b_eff"))
        grid.close()
    assert np.array_equal(out[0], out[1])
    assert not np.array_equal(out[0], before)
    q = np.rint((np.stack([before, out[0]]) - datum) * 2.0 ** k).astype(np.int64)
    assert q[0].sum() == q[1].sum()
    assert int(net.status.item()) == 0
