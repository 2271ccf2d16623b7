"""The weight-gradient kernel at the edges of its bands: widths around a
16-pixel MMA step and a 128-pixel band, heights around the rows of a band, one
and two bands per CTA (more than 148 bands), every channel pair, against the
oracle.  Bound: products of BF16 values are exact in FP32, so an output is off
by at most the roundings of a sum of n terms, n 2^-24 of the magnitudes' sum."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import learned as L  # noqa: E402
from soilb200 import learned as ln  # noqa: E402

pytestmark = pytest.mark.gpu


def _bf16(rng, *shape):
    return torch.as_tensor(rng.normal(size=shape)).to(torch.bfloat16)


@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 32), (32, 16), (32, 32)])
@pytest.mark.parametrize("b,h,w,rows", [(1, 1, 1, 16), (1, 3, 15, 2), (2, 5, 16, 1), (1, 9, 17, 4),
                                        (2, 17, 127, 16), (1, 18, 128, 5), (1, 6, 129, 3),
                                        (3, 34, 260, 16), (40, 16, 24, 4), (149, 4, 8, 16)])
def test_wgrad_band_edges(b, h, w, rows, cin, cout):
    rng = np.random.default_rng(b * 1000 + h * 10 + w)
    x, g = _bf16(rng, b, h, w, cin), _bf16(rng, b, h, w, cout)
    got = ln.wgrad(x.cuda(), g.cuda(), cin, cout, rows=rows).cpu().numpy().astype(np.float64)
    xd, gd = x.double().numpy(), g.double().numpy()
    want = L.conv3x3_wgrad(xd, gd)
    size = L.conv3x3_wgrad(np.abs(xd), np.abs(gd))
    assert np.all(np.abs(got - want) <= b * h * w * 2.0 ** -24 * size + 2.0 ** -24 * np.abs(want))


def test_packed_weights_are_the_gathered_ones():
    net = ln.ReposeNet(seed=4)
    for w in net.weights:  # padded channels too, and values that round
        w.copy_(torch.randn(w.shape, generator=torch.Generator().manual_seed(w.numel())))
    for li, (ci, co) in enumerate(ln.LAYERS):
        w = net.weights[li].cpu()
        fwd = w.reshape(-1)[torch.as_tensor(ln.pack_index(ci, co))].to(torch.bfloat16)
        bwd = ln.flip_transpose(w).reshape(-1)[torch.as_tensor(ln.pack_index(co, ci))]
        assert torch.equal(net.packed()[li].cpu(), fwd)
        assert torch.equal(net.packed_backward()[li].cpu(), bwd.to(torch.bfloat16))
    # weights of another form take the gather
    want = net.packed()
    net.weights = [w.double() for w in net.weights]
    assert all(torch.equal(g, w) for g, w in zip(net.packed(), want))


@pytest.mark.parametrize("rot", ["0", "1"])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("cin,cout", [(16, 16), (32, 16), (16, 32), (32, 32)])
@pytest.mark.parametrize("w", [1, 3, 4, 127, 130])
def test_bf16_rows_are_the_rounded_f32_rows(monkeypatch, w, cin, cout, masked, rot):
    """The exchanged 16-byte pieces of a BF16 row against the FP32 output, which
    each thread writes for its own pixel: the same values, rounded."""
    monkeypatch.setenv("SOILB200_CONV_ROT", rot)
    rng = np.random.default_rng(w + cin + 2 * cout)
    x, m = _bf16(rng, 2, 5, w, cin).cuda(), _bf16(rng, 2, 5, w, cout).cuda()
    wpk = _bf16(rng, 9 * cin * cout).cuda()
    mask = m if masked else None
    for relu in (False, True):
        f32 = ln.conv(x, wpk, cin, cout, relu=relu, out_f32=True, mask=mask)
        out = ln.conv(x, wpk, cin, cout, relu=relu, mask=mask)
        assert torch.equal(out, f32.to(torch.bfloat16))
        if masked:
            assert not torch.any(out[~(m > 0)])
