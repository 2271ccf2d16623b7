"""Proposals and sweeps go to the grid's stream, so the grid's device has to be the
current one at each of their calls, whichever it was before (a second GPU's grid in a
process that works on the first).  On fakes of torch and of the library."""

import contextlib
from types import SimpleNamespace

import pytest

from soilb200 import learned


@pytest.mark.parametrize("fused", [True, False])
def test_proposals_run_on_the_grids_device(monkeypatch, fused):
    current, seen = [0], []

    @contextlib.contextmanager
    def device(index):
        before, current[0] = current[0], index
        yield
        current[0] = before

    def call(*_):
        seen.append(current[0])
        return 0

    fake = SimpleNamespace(cuda=SimpleNamespace(device=device, stream=lambda s: device(s.device)))
    monkeypatch.setattr(learned, "_torch", lambda: fake)
    monkeypatch.setattr(learned._lib, "load", lambda: SimpleNamespace(
        sb_learned_propose=call, sb_learned_features=call, sb_learned_apply=call,
        sb_relax_sweeps=call, sb_relax_full=call))
    buffer = SimpleNamespace(data_ptr=lambda: 0)
    monkeypatch.setattr(learned, "network_forward", lambda *a, **k: (call(), buffer))
    lr = object.__new__(learned.LearnedRelaxation)
    lr.fused, lr.tan_crit = fused, 0.7
    lr.grid = SimpleNamespace(ctx=None, _ctx=None)
    lr.net = SimpleNamespace(device=1, status=buffer)
    lr._feat = lr._flux = lr._tq = buffer
    lr._packed, lr._stream = [buffer] * 4, 0
    lr._torch_stream = SimpleNamespace(device=1)
    lr.propose(3)
    assert seen == [1] * (3 if fused else 9)
    lr.relax(1e-4, scales=(1.0, 0.5), rounds=2, plain_between=5, spacing=(0.05, 0.05))
    assert seen == [1] * (3 + 5 if fused else 9 + 9)  # two rounds, two sweep calls, the last
    assert current == [0]
