"""The weight gradient on inputs beside the ordinary: tensors that do not start
on 16 bytes (cut out of a larger buffer), and an infinite value, which reaches
the outputs that it is a term of and no other."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from soilb200 import learned as ln  # noqa: E402

pytestmark = pytest.mark.gpu


def _at(t, offset: int):
    """A copy of t that starts ``offset`` elements into its buffer."""
    buf = torch.empty(t.numel() + offset, dtype=t.dtype, device=t.device)
    out = buf[offset:].view(t.shape)
    out.copy_(t)
    assert out.data_ptr() % 16 == 2 * offset % 16
    return out


@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 32), (32, 16)])
@pytest.mark.parametrize("shift_x,shift_g", [(1, 0), (0, 3), (4, 7), (8, 8)])
def test_any_start_gives_the_same_gradient(cin, cout, shift_x, shift_g):
    """The same values in the same order: equal bits."""
    gen = torch.Generator().manual_seed(cin + cout)
    for b, h, w in ((1, 1, 1), (2, 5, 17), (1, 9, 131)):
        x = torch.randn(b, h, w, cin, generator=gen).to(torch.bfloat16).cuda()
        g = torch.randn(b, h, w, cout, generator=gen).to(torch.bfloat16).cuda()
        want = ln.wgrad(x, g, cin, cout, rows=4)
        got = ln.wgrad(_at(x, shift_x), _at(g, shift_g), cin, cout, rows=4)
        assert torch.equal(got, want)


def _wgrad_terms(x, g):
    """dW and the sum of its terms' magnitudes, from the terms that exist alone
    (no padding: 0 * inf would be a term)."""
    b, h, w, ci = x.shape
    dw, size = np.zeros((2, 3, 3, ci, g.shape[3]))
    for dy in range(3):
        for dx in range(3):
            y0, y1 = max(0, 1 - dy), min(h, h + 1 - dy)
            x0, x1 = max(0, 1 - dx), min(w, w + 1 - dx)
            xs, gs = x[:, y0 + dy - 1:y1 + dy - 1, x0 + dx - 1:x1 + dx - 1], g[:, y0:y1, x0:x1]
            for c in range(ci):
                t = xs[..., c, None] * gs
                dw[dy, dx, c] = t.sum(axis=(0, 1, 2))
                size[dy, dx, c] = np.abs(t).sum(axis=(0, 1, 2))
    return dw, size


@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 32), (32, 16), (32, 32)])
@pytest.mark.parametrize("h,rows", [(1, 16), (3, 16), (5, 1), (7, 3), (9, 5), (8, 3), (6, 16)])
def test_an_infinite_input_stays_in_its_outputs(h, rows, cin, cout):
    """Bound as for finite inputs: the roundings of a sum of n terms, n 2^-24 of
    the magnitudes' sum."""
    rng = np.random.default_rng(h * 100 + rows)
    g = torch.as_tensor(rng.normal(size=(1, h, 16, cout))).to(torch.bfloat16)
    g[g == 0] = 1.0
    for row in range(h):
        x = torch.as_tensor(rng.normal(size=(1, h, 16, cin))).to(torch.bfloat16)
        x[0, row, 7, 5] = float("inf")
        got = ln.wgrad(x.cuda(), g.cuda(), cin, cout, rows=rows).cpu().numpy().astype(np.float64)
        want, size = _wgrad_terms(x.double().numpy(), g.double().numpy())
        finite = np.isfinite(want)
        assert finite.any() and not np.isnan(want).any()
        assert np.array_equal(got[~finite], want[~finite]), row
        got, want, size = got[finite], want[finite], size[finite]
        assert np.all(np.abs(got - want)
                      <= h * 16 * 2.0 ** -24 * size + 2.0 ** -24 * np.abs(want)), row
