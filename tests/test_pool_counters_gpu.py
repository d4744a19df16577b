"""GPU: the library's memory counters return to where they were once a handle is gone, whatever was built on
it."""
from __future__ import annotations

import gc

import pytest

from _step_cases import template

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _live():
    from conatus_gb300 import core
    gc.collect()
    torch.cuda.synchronize()
    return core.pool_stats()[0]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_nothing_counted_after_a_factor_set(precision, cuda_lib):
    from conatus_gb300 import autotune
    from conatus_gb300.ivp import DeviceProblem
    dev = DeviceProblem(template("rb_nz16").instantiate([32]), precision)
    dev.autotune = False
    n0 = _live()
    fs = dev.factor(1.5e3, 1.0)
    for sched in (0, min(autotune.windowed_schedules()), min(autotune.partitioned_schedules()),
                  *autotune.scheduled_schedules()):
        autotune.apply(fs, sched)
    assert _live() > n0
    dev._factors.clear()
    del fs
    assert _live() == n0
