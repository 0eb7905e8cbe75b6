"""Smoothed fields share one transform plan per size, whose spectrum lives from the first step of a call to the
second: calls from several threads and streams must not come between (a stand-in plan, no GPU)."""
import contextlib
import threading
import time
import types

import pytest

from conftest import module

torch = pytest.importorskip("torch")


class FakeStream:
    cuda_stream = 0

    def __init__(self):
        self.waits = []

    def wait_event(self, e):
        self.waits.append(e.last)


class FakeEvent:
    last = None

    def record(self, stream):
        self.last = stream


class FakePlan:
    """Keeps the last forward()ed box, as the plan keeps its spectrum."""
    made = 0

    def __init__(self, n, box_len, max_radii=1, device=None):
        time.sleep(0.02)
        FakePlan.made += 1
        self.handle, self.box, self.mixed = None, None, 0
        self.lib = types.SimpleNamespace(es_smooth=self.smooth)

    def forward(self, delta):
        self.box = (threading.get_ident(), delta)
        time.sleep(0.005)

    def smooth(self, handle, radii, count, out, stream):
        self.mixed += self.box[0] != threading.get_ident()
        return 0


@pytest.fixture
def shared(monkeypatch):
    sg = module("surrogate")
    current = threading.local()
    monkeypatch.setattr(module("engine"), "ExcursionSetPlan", FakePlan)
    monkeypatch.setattr(sg, "_smooth_plans", {})
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: current.__dict__.setdefault("stream", FakeStream()))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: getattr(current, "capturing", False))
    monkeypatch.setattr(torch.cuda, "Event", FakeEvent)
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    FakePlan.made = 0
    return sg, current


def test_threads_do_not_come_between_the_steps_of_a_call(shared):
    sg, _ = shared
    done = []

    def work():
        for _ in range(5):
            sg.smoothed_fields(torch.zeros(4, 4, 4), (1.0,))
        done.append(1)

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(done) == 4 and FakePlan.made == 1
    plan = next(iter(sg._smooth_plans.values()))
    assert getattr(plan, "plan", plan).mixed == 0


def test_another_stream_waits_for_the_last_call(shared):
    sg, current = shared
    d = torch.zeros(4, 4, 4)
    a, b = FakeStream(), FakeStream()
    for s in (a, a, b, a):
        current.stream = s
        sg.smoothed_fields(d, (1.0,))
    assert b.waits == [a] and a.waits == [b]
    # a call that is being captured neither waits for events of uncaptured work nor leaves one
    current.stream, current.capturing = b, True
    sg.smoothed_fields(d, (1.0,))
    current.stream, current.capturing = a, False
    sg.smoothed_fields(d, (1.0,))
    assert b.waits == [a] and a.waits == [b]
