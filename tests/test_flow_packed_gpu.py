"""GPU: the operations of several handles made side by side: batches small enough to stay laid out at their
most, larger ones packed, larger ones counted first (host-built handles); all handles or none."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

from _step_cases import template

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("share", [True, False])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_packed_operations(share, precision, rng, cuda_lib):
    """The channel's buckets of 1, 23, 23 and 529 systems (one or two of the last): schedule 0's bits."""
    from conatus_gb300 import autotune
    from conatus_gb300.ivp import DeviceProblem
    dev = DeviceProblem(template("channel_ny129").instantiate([48, 48]), precision, share=share)
    dev.autotune = False
    fs = dev.factor(1.5e3, 1.0)
    assert max(dev.nsys) * 400 * (522 + 64) > 64 << 20
    b = dev.zeros()
    b.copy_(torch.as_tensor(rng.standard_normal(dev.n_total) + 1j * rng.standard_normal(dev.n_total)))

    def solve(sched):
        autotune.apply(fs, sched)
        x = dev.zeros()
        dev._batch_call(fs, list(range(len(fs))), b, x, None, int(precision == "fp32"), 0, None)
        torch.cuda.synchronize()
        return x
    like32, like16 = autotune.scheduled_schedules()
    assert torch.equal(solve(like16), solve(0))
    if not share:
        split = min(autotune.split_schedules())
        assert torch.equal(solve(like32), solve(split))


def test_counted_operations(rng, cuda_lib):
    """A host-built batch above 64 MB of operations at their most, below its limit."""
    from conatus_gb300 import core
    n, batch = 200, 700
    assert 64 << 20 < batch * 400 * (n + 64) < 1 << 30
    mats = []
    for _ in range(batch):
        A = sp.diags([rng.standard_normal(n - 2), 4 + rng.standard_normal(n), rng.standard_normal(n - 4)], [-2, 0, 4],
                     format="lil")
        A[0] = rng.standard_normal(n)
        mats.append(A.tocsr().astype(complex))
    live = core.pool_stats()[0]
    h = core.cuda.BandedBatchZ([(n, A.indptr, A.indices, A.data) for A in mats], [0])
    assert core.pool_stats()[0] - live > batch * n * 16 * 3
    b = rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))
    x = torch.as_tensor(b, device="cuda")
    h.solve_ptr(x.data_ptr(), batch, n)
    for A, bi, xi in zip(mats, b, x.cpu().numpy()):
        D = A.toarray()
        ref = np.linalg.solve(D, bi)
        assert np.linalg.norm(xi - ref) <= 4 * n * EPS * np.linalg.cond(D) * np.linalg.norm(ref)


def test_all_or_none(rng, cuda_lib):
    """A shared pair among the handles refuses the 32-lane schedule: the others keep theirs too."""
    from conatus_gb300 import autotune
    from conatus_gb300._lib import call
    from conatus_gb300.ivp import DeviceProblem
    dev = DeviceProblem(template("channel_ny17").instantiate([8, 8]), "fp64", share=True)
    dev.autotune = False
    fs = dev.factor(1.5e3, 1.0)
    assert dev.shared
    b = dev.zeros()
    b.copy_(torch.as_tensor(rng.standard_normal(dev.n_total) + 1j * rng.standard_normal(dev.n_total)))

    def solve():
        x = dev.zeros()
        dev.solve(1.5e3, 1.0, b, x)
        torch.cuda.synchronize()
        return x
    own = [h.h.value for h in fs if h.h is not None]
    hs = (ctypes.c_void_p * len(own))(*own)
    like32, like16 = autotune.scheduled_schedules()
    for before in (0, like16):
        autotune.apply(fs, before)
        ref = solve()
        for refused in (like32, min(autotune.partitioned_schedules()), 99):
            with pytest.raises(ValueError):
                call("cng_banded_set_schedule_all", len(own), hs, refused)
            assert torch.equal(solve(), ref)
    with pytest.raises(ValueError):
        call("cng_banded_set_schedule_all", 0, hs, 0)
    with pytest.raises(ValueError):
        call("cng_banded_set_schedule_all", 1, (ctypes.c_void_p * 1)(None), 0)
