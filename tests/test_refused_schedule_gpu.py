"""GPU: a schedule that a handle refuses leaves it with the one it has: the next solve gives the same bits."""
from __future__ import annotations

import numpy as np
import pytest

from _step_cases import template

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _solver(tname, sizes, share, rng, precision="fp64"):
    from conatus_gb300 import autotune
    from conatus_gb300.ivp import DeviceProblem
    dev = DeviceProblem(template(tname).instantiate(sizes), precision, share=share)
    fs = dev.factor(1.5e3, 1.0)
    b = dev.zeros()
    b.copy_(torch.as_tensor(rng.standard_normal(dev.n_total) + 1j * rng.standard_normal(dev.n_total)))

    def solve():
        x = dev.zeros()
        dev.solve(1.5e3, 1.0, b, x)
        torch.cuda.synchronize()
        return x
    return autotune, dev, fs, solve


def _refused(fs, sched):
    from conatus_gb300._lib import call
    n = 0
    for h in fs:
        if h.h is not None:
            try:
                call("cng_banded_set_schedule", h.h, sched)
            except ValueError:
                n += 1
    return n


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_shared_pairs_keep_the_scheduled_solve(precision, rng, cuda_lib):
    """A shared pair refuses the partitioned schedule and the 32-lane scheduled solve."""
    autotune, dev, fs, solve = _solver("channel_ny17", [8, 8], True, rng, precision)
    assert dev.shared
    only = [h for h in fs if h.h is not None and any(j == fs.index(h) for j in dev.shared.values())]
    like32, like16 = autotune.scheduled_schedules()
    autotune.apply(fs, like16)                     # not what an earlier test timed
    ref = solve()
    for sched in (min(autotune.partitioned_schedules()), like32):
        assert _refused(only, sched) == len(only) > 0
        assert torch.equal(solve(), ref)


def test_the_windowed_scratch_stays_too(rng, cuda_lib):
    autotune, dev, fs, solve = _solver("channel_ny17", [8, 8], True, rng)
    only = [h for h in fs if h.h is not None and any(j == fs.index(h) for j in dev.shared.values())]
    autotune.apply(fs, min(autotune.windowed_schedules()))
    ref = solve()
    assert _refused(only, min(autotune.partitioned_schedules())) == len(only) > 0
    assert torch.equal(solve(), ref)


def test_host_built_handles_keep_their_operations(rng, cuda_lib):
    """A handle of host matrices refuses schedules it has no streams for and keeps its solve."""
    import scipy.sparse as sp
    from conatus_gb300 import core
    from conatus_gb300._lib import call
    n = 40
    A = sp.diags([rng.standard_normal(n - 1), 4 + rng.standard_normal(n), rng.standard_normal(n - 1)], [-1, 0, 1]).tocsr()
    h = core.cuda.BandedBatchZ([(n, A.indptr, A.indices, A.data.astype(complex))] * 3, [])
    b = torch.as_tensor(rng.standard_normal((3, n)) + 1j * rng.standard_normal((3, n)), device="cuda")
    x, y = torch.empty_like(b), torch.empty_like(b)
    h.solve_mapped_ptr(b.data_ptr(), 0, x.data_ptr(), 0)
    live = core.pool_stats()[0]
    for sched in (0, 12, 99):
        with pytest.raises(ValueError):
            call("cng_banded_set_schedule", h._h.h, sched)
    assert core.pool_stats()[0] == live
    h.solve_mapped_ptr(b.data_ptr(), 0, y.data_ptr(), 0)
    assert torch.equal(x, y)
    assert np.allclose((A @ x.cpu().numpy().T).T, b.cpu().numpy(), atol=1e-10)
