"""Closed initial conditions make no new plan (stand-in plans, no GPU)."""
import pytest

from conftest import module

torch = pytest.importorskip("torch")


class FakePlan:
    made = 0

    def __init__(self, *a, **k):
        FakePlan.made += 1
        self.closed = False

    def close(self):
        self.closed = True


def test_plan_is_made_once_and_not_after_close(monkeypatch):
    monkeypatch.setattr(module("engine"), "ExcursionSetPlan", FakePlan)
    ini = module("initial")
    ic = ini.InitialConditions.__new__(ini.InitialConditions)
    ic.dim, ic.box_len, ic.device = 32, 50.0, None
    ic._plan, ic._fft, ic._small = None, FakePlan(), None
    FakePlan.made = 0
    full = ic.plan
    assert ic.plan is full and FakePlan.made == 1
    fft = ic._fft
    ic.close()
    assert full.closed and fft.closed
    assert ic.plan is None and FakePlan.made == 1
    ic.close()
