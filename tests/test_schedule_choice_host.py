"""CPU: which solve schedule a new factor set gets: a scheduled solve where the systems take it, the
fastest timed one otherwise, the fixed one where the environment fixes it."""
from __future__ import annotations

import types

import pytest

from conatus_gb300 import autotune


@pytest.fixture
def applied(monkeypatch):
    out = []
    monkeypatch.setattr(autotune, "scheduled_schedules", lambda: (19, 20))
    monkeypatch.setattr(autotune, "tune_solve", lambda dev, key, fs, stream=None: {7: 1.0})
    monkeypatch.setattr(autotune, "_CACHE", {})
    monkeypatch.delenv("CONATUS_GB300_SOLVE_SCHEDULE", raising=False)

    def apply(fs, sched):
        out.append(sched)
        if fs[0].refuse:
            raise ValueError("not real up to powers of i")
    monkeypatch.setattr(autotune, "apply", apply)
    return out


def _case(d, refuse=False):
    h = types.SimpleNamespace(batch=4, n=262, rank=6, kl=9, ku=22, refuse=refuse, h=1)
    return types.SimpleNamespace(d=d, precision="fp64", shared={}), [h]


@pytest.mark.parametrize("d,want", [(0, 19), (1, 20), (2, 20)])
def test_the_scheduled_solve_where_it_applies(applied, d, want):
    dev, fs = _case(d)
    assert autotune.choose_solve(dev, (1.0, 0.5), fs) == {want: None} and applied == [want]


def test_timed_where_it_is_refused(applied, monkeypatch):
    dev, fs = _case(1, refuse=True)
    assert autotune.choose_solve(dev, (1.0, 0.5), fs) == {7: 1.0} and applied == [20]
    autotune._CACHE[autotune._signature(dev, fs)] = (7, {7: 1.0})        # known: not tried again
    assert autotune.choose_solve(dev, (1.0, 0.5), fs) == {7: 1.0} and applied == [20]
    dev, fs = _case(1)
    monkeypatch.setenv("CONATUS_GB300_SOLVE_SCHEDULE", "3")
    autotune._CACHE.clear()
    assert autotune.choose_solve(dev, (1.0, 0.5), fs) == {7: 1.0} and applied == [20]
