"""CPU: the planned bytes of a factor set hold the compact streams or the scheduled solve's operations,
whichever are larger, not both: what a memory budget admits stays what it was with streams alone."""
from __future__ import annotations

import pytest

from conatus_gb300 import memory, workloads as W


@pytest.mark.parametrize("precision,streams_alone", [("fp64", 36.238e9), ("fp32", 44.346e9)])
def test_the_headline_channel(precision, streams_alone):
    P = W.problem("channel")
    assert memory.plan_ivp(P, W.CONFIGS["channel"]["scheme"], precision)["total"] <= streams_alone


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_at_least_the_operations(precision):
    """400 bytes per column and system, two thirds of that again for their FP32 copies."""
    P = W.problem("rayleigh_benard")
    parts = memory.plan_ivp(P, "SBDF2", precision, factor_sets=1)
    least = sum(ns * 400 * b.n * (5 if precision == "fp32" else 3) // 3 for ns, b in zip(P.nsys, P.tpl.buckets))
    assert parts["factors"] >= least
