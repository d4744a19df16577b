"""CPU: a new factor set on a device without room for the scheduled solve's operations: the schedules that
need none are timed, and candidates that do not fit are passed over like those that do not apply."""
from __future__ import annotations

import types

import pytest

from conatus_gb300 import autotune
from conatus_gb300.errors import CudaError, check_status

NO_ROOM = "cudaMalloc of 921600000 bytes failed: out of memory"


def _case():
    h = types.SimpleNamespace(batch=4, n=262, rank=6, kl=9, ku=22, h=1, schedule=None)
    return types.SimpleNamespace(d=1, precision="fp64", shared={}), [h]


def test_no_room_for_the_operations(monkeypatch):
    monkeypatch.setattr(autotune, "scheduled_schedules", lambda: (19, 20))
    monkeypatch.setattr(autotune, "tune_solve", lambda dev, key, fs, stream=None: {7: 1.0})
    monkeypatch.setattr(autotune, "_CACHE", {})
    monkeypatch.delenv("CONATUS_GB300_SOLVE_SCHEDULE", raising=False)

    def apply(fs, sched):
        check_status(3, NO_ROOM, "cng_banded_set_schedule")
    monkeypatch.setattr(autotune, "apply", apply)
    dev, fs = _case()
    assert autotune.choose_solve(dev, (1.0, 0.5), fs) == {7: 1.0}


def test_other_failures_are_raised(monkeypatch):
    monkeypatch.setattr(autotune, "scheduled_schedules", lambda: (19, 20))
    monkeypatch.setattr(autotune, "_CACHE", {})
    monkeypatch.delenv("CONATUS_GB300_SOLVE_SCHEDULE", raising=False)

    def apply(fs, sched):
        check_status(3, "k_flow_build: invalid device function", "cng_banded_set_schedule")
    monkeypatch.setattr(autotune, "apply", apply)
    dev, fs = _case()
    with pytest.raises(CudaError, match="invalid device function"):
        autotune.choose_solve(dev, (1.0, 0.5), fs)


def test_the_error_is_still_a_cuda_error():
    with pytest.raises(CudaError, match="cng_banded_create_csr: cudaMalloc of"):
        check_status(3, NO_ROOM, "cng_banded_create_csr")


def test_timed_candidates_without_room(monkeypatch):
    """tune_solve with a candidate that does not fit beside the others."""
    import conatus_gb300.ivp as ivp
    t = {"now": 0.0}

    class Event:
        def __init__(self, enable_timing=False):
            self.t = 0.0

        def record(self, stream=None):
            self.t = t["now"]

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
    monkeypatch.setattr(autotune, "schedules", lambda: [0, 1, 2])
    monkeypatch.setattr(autotune, "partitioned_schedules", lambda: set())
    monkeypatch.setattr(autotune, "_CACHE", {})
    monkeypatch.delenv("CONATUS_GB300_SOLVE_SCHEDULE", raising=False)

    def apply(fs, sched):
        if sched == 1:
            check_status(3, NO_ROOM, "cng_banded_set_schedule")
        fs[0].schedule = sched
    monkeypatch.setattr(autotune, "apply", apply)
    dev, fs = _case()
    dev.zeros = lambda: types.SimpleNamespace(fill_=lambda v: None)

    def solve(fs, a, b, rhs, out, st):
        t["now"] += 3.0 - fs[0].schedule
    dev._solve_with = solve
    assert autotune.tune_solve(dev, (1.0, 0.5), fs) == {0: 3.0, 2: 1.0} and fs[0].schedule == 2
