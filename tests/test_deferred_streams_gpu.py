"""GPU: the compact streams of a factor set are made when a schedule reads them: none beside the scheduled
solve, and every schedule set later solves with the bits of a factor set whose streams were there first."""
from __future__ import annotations

import pytest

from _step_cases import template

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

A, B = 1.5e3, 1.0


def _problem(tname, sizes, share, precision, autotune):
    from conatus_gb300.ivp import DeviceProblem
    dev = DeviceProblem(template(tname).instantiate(sizes), precision, share=share)
    dev.autotune = autotune
    return dev


def _live():
    from conatus_gb300 import core
    torch.cuda.synchronize()
    return core.pool_stats()[0]


@pytest.fixture
def fresh(monkeypatch):
    from conatus_gb300 import autotune
    monkeypatch.setattr(autotune, "_CACHE", {})
    monkeypatch.delenv("CONATUS_GB300_SOLVE_SCHEDULE", raising=False)
    return autotune


@pytest.mark.parametrize("tname,sizes,share", [("rb_nz16", [32], True), ("channel_ny17", [14, 6], True),
                                               ("channel_ny17", [8, 8], False), ("burgers_n128", None, True)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_every_schedule_after_the_scheduled_solve(tname, sizes, share, precision, fresh, rng, cuda_lib):
    dev, eager = (_problem(tname, sizes, share, precision, a) for a in (True, False))
    fs, es = dev.factor(A, B), eager.factor(A, B)
    flow = fresh.scheduled_schedules()
    assert all(h.schedule in flow for h in fs if h.h is not None)
    b = dev.zeros()
    b.copy_(torch.as_tensor(rng.standard_normal(dev.n_total) + 1j * rng.standard_normal(dev.n_total)))

    def solve(d):
        x = d.zeros()
        d.solve(A, B, b, x)
        torch.cuda.synchronize()
        return x
    for h in es:
        if h.h is not None:
            h.schedule = 0
    first = solve(dev)
    part, split = fresh.partitioned_schedules(), fresh.split_schedules()
    for sched in [s for s in fresh.schedules() if s not in part and not (dev.shared and (s < 0 or s in split))]:
        fresh.apply(fs, sched)
        fresh.apply(es, sched)
        assert torch.equal(solve(dev), solve(eager)), sched
    fresh.apply(fs, flow[1] if dev.d else flow[0])
    assert torch.equal(solve(dev), first)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_no_streams_beside_the_scheduled_solve(precision, fresh, cuda_lib):
    """The factor set with its operations against one whose streams were made first and stay: less by the
    streams, which hold a diagonal entry and a pivot per column and system at least."""
    n0 = _live()
    dev, eager = (_problem("channel_ny129", [24, 24], True, precision, a) for a in (True, False))
    n1 = _live()
    fs = dev.factor(A, B)
    held = _live() - n1
    n2 = _live()
    es = eager.factor(A, B)
    fresh.apply(es, 0)
    streams = _live() - n2
    like16 = fresh.scheduled_schedules()[1]
    fresh.apply(es, like16)
    both = _live() - n2
    least = sum(h.batch * h.n * 20 for h in fs if h.h is not None)
    assert held <= both - least, (held, both, least)
    fresh.apply(fs, 0)
    assert _live() - n1 == streams + both          # the operations go, the streams come
    fresh.apply(fs, like16)
    assert _live() - n1 == held + both
    del dev, fs, eager, es
    import gc
    gc.collect()
    assert _live() == n0


def test_buckets_of_different_schedules(fresh, rng, cuda_lib):
    """Schedule 0 solves buckets whose schedules differ, streams or not."""
    dev = _problem("channel_ny17", [14, 6], True, "fp64", True)
    fs = dev.factor(A, B)
    b = dev.zeros()
    b.copy_(torch.as_tensor(rng.standard_normal(dev.n_total) + 1j * rng.standard_normal(dev.n_total)))
    x, y = dev.zeros(), dev.zeros()
    dev.solve(A, B, b, x)
    fresh.apply(fs[:1], 0)
    dev.solve(A, B, b, y)
    torch.cuda.synchronize()
    assert torch.equal(x, y)                       # the scheduled solve has schedule 0's bits


def test_a_plan_of_the_memory(fresh, cuda_lib):
    """What a solver holds stays within the planned bytes of the larger of both."""
    from conatus_gb300 import memory
    P = template("channel_ny129").instantiate([24, 24])
    from conatus_gb300.ivp import IVPSolver
    from conatus_gb300 import workloads as W
    for precision in ("fp64", "fp32"):
        n0, t0 = _live(), torch.cuda.memory_allocated()
        s = IVPSolver(P, scheme="SBDF3", dt=5e-3, precision=precision, factor_sets=1)
        s.set_state(W.initial_state("channel", P, seed=0))
        s.run(4)
        held = _live() - n0 + torch.cuda.memory_allocated() - t0
        plan = memory.plan_ivp(P, "SBDF3", precision, factor_sets=1)["total"]
        assert held <= plan + (8 << 20), (precision, held, plan)
        del s
        import gc
        gc.collect()
