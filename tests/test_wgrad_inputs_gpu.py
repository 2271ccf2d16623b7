"""The weight gradient on inputs beside the ordinary: tensors that do not start
on 16 bytes (cut out of a larger buffer)."""

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
