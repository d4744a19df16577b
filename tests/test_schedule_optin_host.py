"""CPU: a problem that opts into the partitioned solve has it timed beside every other schedule, the
scheduled solve among them; one that does not gets the scheduled solve untimed."""
from __future__ import annotations

import types

import pytest

from conatus_gb300 import autotune

TIMES = {-1: 9.0, 0: 4.0, 11: 2.0, 19: 3.0, 20: 3.5}


@pytest.fixture
def timed(monkeypatch):
    import conatus_gb300.ivp as ivp
    clock = {"t": 0.0}

    class Event:
        def __init__(self, enable_timing=False):
            self.t = 0.0

        def record(self, stream=None):
            self.t = clock["t"]

        def synchronize(self):
            pass

        def elapsed_time(self, other):
            return other.t - self.t

    class Ctx:
        def __enter__(self):
            return self

        def __exit__(self, *a):
            return False
    cuda = types.SimpleNamespace(Event=Event, current_stream=lambda: "s", stream=lambda s: Ctx(), ExternalStream=lambda p: p)
    monkeypatch.setattr(ivp, "_torch", lambda: types.SimpleNamespace(cuda=cuda))
    monkeypatch.setattr(autotune, "schedules", lambda: sorted(TIMES))
    monkeypatch.setattr(autotune, "partitioned_schedules", lambda: {11})
    monkeypatch.setattr(autotune, "scheduled_schedules", lambda: (19, 20))
    monkeypatch.setattr(autotune, "_CACHE", {})
    monkeypatch.delenv("CONATUS_GB300_SOLVE_SCHEDULE", raising=False)

    def apply(fs, sched):
        fs[0].schedule = sched
    monkeypatch.setattr(autotune, "apply", apply)

    def case(partitioned, scheduled_ms=None, d=1):
        h = types.SimpleNamespace(batch=127, n=262, rank=6, kl=9, ku=22, h=1, schedule=None)
        dev = types.SimpleNamespace(d=d, precision="fp64", shared={}, partitioned=partitioned,
                                    zeros=lambda: types.SimpleNamespace(fill_=lambda v: None))

        def solve(fs, a, b, rhs, out, st):
            s = fs[0].schedule
            clock["t"] += scheduled_ms if scheduled_ms is not None and s in (19, 20) else TIMES[s]
        dev._solve_with = solve
        return dev, [h]
    return case


def test_opted_in_it_is_timed(timed):
    dev, fs = timed(True)
    times = autotune.choose_solve(dev, (1.0, 0.5), fs)
    assert set(times) == set(TIMES) and fs[0].schedule == 11


def test_the_faster_one_is_kept(timed):
    dev, fs = timed(True, scheduled_ms=1.0)
    times = autotune.choose_solve(dev, (1.0, 0.5), fs)
    assert 11 in times and fs[0].schedule in (19, 20)


def test_not_opted_in(timed):
    dev, fs = timed(False)
    assert autotune.choose_solve(dev, (1.0, 0.5), fs) == {20: None} and fs[0].schedule == 20
