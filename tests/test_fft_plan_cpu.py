"""Transform plans that find no device memory: the engine's error, as for any other plan (no GPU: the allocation
fails in a stand-in)."""
import contextlib
import types

import pytest

from conftest import module

torch = pytest.importorskip("torch")


def test_no_memory_is_the_engines_error(monkeypatch):
    eng, _lib = module("engine"), module("_lib")

    def refuse(*a, **k):
        raise torch.OutOfMemoryError("CUDA out of memory")

    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    monkeypatch.setattr(_lib, "load", lambda: types.SimpleNamespace(es_fft_plan_bytes=lambda n, s: 1 << 50))
    monkeypatch.setattr(torch, "empty", refuse)
    with pytest.raises(_lib.EngineError) as e:
        eng.FftPlan(512, 300.0)
    assert e.value.code == _lib.ES_E_NOMEM
