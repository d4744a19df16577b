"""GPU: host-built handles whose operations fit, told by the memory they hold, solve like the dense solver:
bands wider than a warp, many border rows, single columns, rows in any order. And the ones whose operations
do not fit hold none and solve too."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps
BATCH = 3


def _system(rng, n, diags, r, filled, complex_, p, q):
    A = np.zeros((n, n))
    for d in diags:
        A += np.diag(rng.standard_normal(n - abs(d)), d)
    A += 6.0 * np.eye(n)
    A[:r] = rng.standard_normal((r, n)) * (rng.random((r, n)) < filled)
    A[np.arange(r), np.arange(r)] += 6.0
    return A * np.where(p[:, None] == q[None], 1, np.where(p[:, None] > q[None], 1j, -1j)) if complex_ else A


def _solve(rng, n, diags, r, filled, complex_):
    from conatus_gb300 import core
    p, q = rng.integers(0, 2, n), rng.integers(0, 2, n)
    p[:r] = q[:r]
    mats = [_system(rng, n, diags, r, filled, complex_, p, q) for _ in range(BATCH)]
    csr = [sp.csr_matrix(A) for A in mats]
    live = core.pool_stats()[0]
    cls = core.cuda.BandedBatchZ if complex_ else core.cuda.BandedBatchD
    h = cls([(n, C.indptr, C.indices, C.data) for C in csr], list(range(r)))
    e = 16 if complex_ else 8
    at_least = lambda size: max(size, 16)
    factors = sum(at_least(s) for s in (BATCH * n * h._h.ldab * e, BATCH * n * 4, BATCH * r * n * e, BATCH * r * n * e,
                                        BATCH * r * r * e, BATCH * r * 4, n * 4, BATCH * 4, BATCH * 8))
    held = core.pool_stats()[0] - live - factors
    b = rng.standard_normal((BATCH, n)) + (1j * rng.standard_normal((BATCH, n)) if complex_ else 0)
    x = torch.as_tensor(b, device="cuda")
    h.solve_ptr(x.data_ptr(), BATCH, n)
    for A, bi, xi in zip(mats, b, x.cpu().numpy()):
        ref = np.linalg.solve(A, bi)
        assert np.linalg.norm(xi - ref) <= 4 * n * EPS * np.linalg.cond(A) * np.linalg.norm(ref)
    return held


@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("n,diags,r,filled", [
    (1, (), 0, 0), (2, (-1,), 0, 0), (2, (), 2, 1.0), (40, (-1, 1), 0, 0), (33, (-1, 1), 1, 1.0),
    (120, (-33, -2), 0, 0), (120, (5, 40), 0, 0), (100, (-40, 40), 2, 0.1), (300, (-34, -1), 3, 0.2),
    (160, (-2, 2), 12, 0.1), (200, (1,), 20, 0.05)])
def test_taken(n, diags, r, filled, complex_, rng, cuda_lib):
    assert _solve(rng, n, diags, r, filled, complex_) >= BATCH * 6144


@pytest.mark.parametrize("n,diags,r,filled,complex_", [
    (131, (-2, -1, 1, 2), 33, 1.0, True), (131, (-2, -1, 1, 2), 33, 1.0, False),
    (70, tuple(range(-40, 39)), 2, 1.0, True), (70, tuple(range(-40, 39)), 2, 1.0, False)])
def test_too_many_operations(n, diags, r, filled, complex_, rng, cuda_lib):
    assert _solve(rng, n, diags, r, filled, complex_) < BATCH * 6144
