"""The plan cache: threads that ask for plans of one geometry while one of them replaces the plan.

The plans are stand-ins without a library handle; their creation and their closing take as long as
the test says.
"""

from __future__ import annotations

import threading

import pytest

torch = pytest.importorskip("torch")

from jht_b200 import _lib  # noqa: E402

KEY = (8, 12, 0, "fp64")


class FakePlan:
    gate = None  # when set, a new plan waits for it
    fail = False
    closed = 0
    handle = None

    def __init__(self, nside, lmax, spin, precision, max_batch=1, device=None):
        if FakePlan.gate is not None:
            FakePlan.started.set()
            assert FakePlan.gate.wait(30)
        if FakePlan.fail:
            raise MemoryError("no room")
        self.max_batch, self.handle = max_batch, object()

    def set_tuning(self, **knobs):
        pass

    def close(self):
        if self.handle is not None:
            FakePlan.closed += 1
        self.handle = None

    __del__ = close


@pytest.fixture
def cache(monkeypatch):
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(_lib, "Plan", FakePlan)
    monkeypatch.setattr(_lib, "_plans", {})
    FakePlan.gate, FakePlan.fail, FakePlan.closed = None, False, 0
    FakePlan.started = threading.Event()


def _replace_in_a_thread():
    """A thread that asks for a larger batch, stopped inside the new plan's creation."""
    FakePlan.gate = threading.Event()
    t = threading.Thread(target=lambda: _lib.get_plan(*KEY, batch=4))
    t.start()
    assert FakePlan.started.wait(30)
    return t


def test_no_call_gets_a_plan_that_is_being_replaced(cache):
    _lib.get_plan(*KEY, batch=1)
    t = _replace_in_a_thread()
    got = []
    other = threading.Thread(target=lambda: got.append(_lib.get_plan(*KEY, batch=1)))
    other.start()
    other.join(0.5)  # either it waits for the new plan, or it has a plan that is still open
    early = [p.handle for p in got]
    FakePlan.gate.set()
    t.join(30)
    other.join(30)
    assert None not in early
    assert got[0].handle is not None and got[0].max_batch >= 1


def test_a_plan_in_use_stays_open_and_an_unused_one_goes(cache):
    held = _lib.get_plan(*KEY, batch=1)
    t = _replace_in_a_thread()
    FakePlan.gate.set()
    t.join(30)
    assert held.handle is not None and FakePlan.closed == 0  # its launches may still be running
    del held
    assert FakePlan.closed == 1
    assert _lib.get_plan(*KEY, batch=8).max_batch == 8 and FakePlan.closed == 2  # nobody held the plan for 4


def test_a_failed_creation_leaves_no_closed_plan(cache):
    _lib.get_plan(*KEY, batch=1)
    FakePlan.fail = True
    with pytest.raises(MemoryError):
        _lib.get_plan(*KEY, batch=4)
    FakePlan.fail = False
    assert _lib.get_plan(*KEY, batch=1).handle is not None


def test_clearing_the_cache_leaves_a_plan_in_use_open(cache):
    held, _ = _lib.get_plan(*KEY, batch=1), _lib.get_plan(16, 24, 0, "fp64")
    del _
    _lib.clear_plans()
    assert FakePlan.closed == 1 and held.handle is not None
    assert _lib.get_plan(*KEY, batch=1) is not held
    del held
    assert FakePlan.closed == 2
