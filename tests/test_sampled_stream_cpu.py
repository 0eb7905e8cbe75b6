"""Sampled fields of the spectrum a transform plan holds: both plans' workspaces are in use on the calling stream and
must not go back to the allocator before its work there is done (stand-in plans, no GPU)."""
import types

import pytest

from conftest import module

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("own_spectrum", [True, False])
def test_workspaces_are_recorded_on_the_calling_stream(monkeypatch, own_spectrum):
    eng = module("engine")
    recorded = []
    monkeypatch.setattr(eng.FftPlan, "_on", lambda self, stream: recorded.append(self))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: None)
    lib = types.SimpleNamespace(ic_sampled_fields=lambda *a: 0, es_plan_destroy=lambda h: 0)
    plans = []
    for n in (32, 16):
        p = eng.FftPlan.__new__(eng.FftPlan)
        p.lib, p._h, p.device, p.n, p.spectra = lib, 1, torch.device("cpu"), n, 4
        plans.append(p)
    big, small = plans
    half = None if own_spectrum else torch.zeros((32, 32, 17), dtype=torch.complex64)
    outs = eng.sampled_fields(big, half, small, -1, 2, 1.0, 1.0)
    assert [tuple(o.shape) for o in outs] == [(16, 16, 16)] * 2
    assert small in recorded and (big in recorded) == own_spectrum
