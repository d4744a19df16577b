"""GPU: a refactored handle solves with the new values whatever schedule it has, FP64 and FP32, and with
any schedule set after: the bits of a handle made from those values; values that its schedule does not
take are solved by another."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N, R, BATCH = 48, 2, 6


def _pattern(rng):
    A = np.zeros((N, N), bool)
    for d in range(-3, 6):
        A |= np.eye(N, k=d, dtype=bool)
    A[:R] = rng.random((R, N)) < 0.7
    A[np.arange(R), np.arange(R)] = True
    return sp.csr_matrix(A)


def _values(rng, C, phases=True):
    """BATCH sets of values: real up to powers of i (times i in odd rows and in odd columns), or of no such
    form."""
    rows = np.repeat(np.arange(N), np.diff(C.indptr))
    v = rng.standard_normal((BATCH, C.nnz)) + 6.0 * (rows == C.indices)
    if phases:
        v = v * np.where(rows % 2 == 1, 1j, 1.0) * np.where(C.indices % 2 == 1, 1j, 1.0)
    else:
        v = v * np.exp(1j * rng.uniform(0, 6, v.shape))
    return torch.as_tensor(v, device="cuda")


def _handle(C, v, fp32):
    from conatus_gb300._lib import call
    from conatus_gb300.core import _Handle
    h = _Handle.shared(np.complex128, BATCH, N, C.indptr, C.indices, v, list(range(R)))
    if fp32:
        call("cng_banded_make_fp32", h.h, None)
    call("cng_banded_compact", h.h, None)
    return h


def _solve(h, b, fp32):
    from conatus_gb300._lib import call
    x = torch.zeros_like(b)
    V = ctypes.c_void_p * 1
    torch.cuda.synchronize()
    call("cng_banded_solve_batch", 1, V(h.h.value), V(b.data_ptr()), V(x.data_ptr()), int(fp32), 0, None)
    torch.cuda.synchronize()
    return x


def _dense(C, v, b, x, tol):
    for k in range(BATCH):
        A = sp.csr_matrix((v[k].cpu().numpy(), C.indices, C.indptr), shape=(N, N)).toarray()
        ref = np.linalg.solve(A, b[k].cpu().numpy())
        assert np.linalg.norm(x[k].cpu().numpy() - ref) <= tol * np.linalg.cond(A) * np.linalg.norm(ref)


def _kinds():
    return ["band", "default", "split", "windowed", "partitioned", "scheduled 32", "scheduled 16"]


def _number(kind):
    from conatus_gb300 import autotune
    like32, like16 = autotune.scheduled_schedules()
    part = autotune.partitioned_schedules()
    return {"band": -1, "default": 0, "split": min(autotune.split_schedules() - part), "windowed": min(autotune.windowed_schedules()),
            "partitioned": min(part), "scheduled 32": like32, "scheduled 16": like16}[kind]


@pytest.mark.parametrize("kind", _kinds())
@pytest.mark.parametrize("fp32", [False, True])
def test_new_values(kind, fp32, rng, cuda_lib):
    from conatus_gb300._lib import call
    if kind == "partitioned" and fp32:
        pytest.skip("FP64 only")
    C = _pattern(rng)
    v1, v2 = _values(rng, C), _values(rng, C)
    b = torch.as_tensor(rng.standard_normal((BATCH, N)) + 1j * rng.standard_normal((BATCH, N)), device="cuda")
    s = _number(kind)
    fresh, h = _handle(C, v2, fp32), _handle(C, v1, fp32)
    call("cng_banded_set_schedule", fresh.h, s)
    call("cng_banded_set_schedule", h.h, s)
    tol = 4 * N * (1.2e-7 if fp32 else 2.3e-16)
    _dense(C, v1, b, _solve(h, b, fp32), tol)
    h.refactor(v2)
    x = _solve(h, b, fp32)
    assert torch.equal(x, _solve(fresh, b, fp32))
    _dense(C, v2, b, x, tol)
    for other in ("default", "scheduled 16", "split"):
        for g in (h, fresh):
            call("cng_banded_set_schedule", g.h, _number(other))
        assert torch.equal(_solve(h, b, fp32), _solve(fresh, b, fp32)), other


@pytest.mark.parametrize("fp32", [False, True])
def test_values_that_the_scheduled_solve_does_not_take(fp32, rng, cuda_lib):
    from conatus_gb300._lib import call
    C = _pattern(rng)
    h = _handle(C, _values(rng, C), fp32)
    call("cng_banded_set_schedule", h.h, _number("scheduled 16"))
    v2 = _values(rng, C, phases=False)
    h.refactor(v2)
    b = torch.as_tensor(rng.standard_normal((BATCH, N)) + 1j * rng.standard_normal((BATCH, N)), device="cuda")
    _dense(C, v2, b, _solve(h, b, fp32), 4 * N * (1.2e-7 if fp32 else 2.3e-16))
    v3 = _values(rng, C)
    h.refactor(v3)
    _dense(C, v3, b, _solve(h, b, fp32), 4 * N * (1.2e-7 if fp32 else 2.3e-16))
