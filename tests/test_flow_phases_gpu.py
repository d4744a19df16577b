"""GPU: large batches of complex systems whose phases are found on a sample of them: a system outside the
sample with other phases (all rows, one row, one column, one border row, or entries that have none) is
solved like every other."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _mats(rng, batch, n, r, phases):
    """Bordered bands (kl = 2, ku = 3), complex by the phases of rows and columns where there are some."""
    p, q = (rng.integers(0, 2, n), rng.integers(0, 2, n)) if phases else (np.zeros(n, int), np.zeros(n, int))
    p[:r] = q[:r]
    out = []
    for _ in range(batch):
        A = np.zeros((n, n))
        for d in range(-min(2, n - 1), min(3, n - 1) + 1):
            A += np.diag(rng.standard_normal(n - abs(d)), d)
        A += 6.0 * np.eye(n)
        A[:r] = rng.standard_normal((r, n))
        A[np.arange(r), np.arange(r)] += 6.0
        out.append(A * np.where(p[:, None] == q[None], 1, np.where(p[:, None] > q[None], 1j, -1j)))
    return out


def _solve(mats, r, b):
    from conatus_gb300 import core
    csr = [sp.csr_matrix(A) for A in mats]
    h = core.cuda.BandedBatchZ([(A.shape[0], C.indptr, C.indices, C.data.astype(complex)) for A, C in zip(mats, csr)],
                               list(range(r)))
    x = torch.as_tensor(b, device="cuda")
    h.solve_ptr(x.data_ptr(), *b.shape)
    return x.cpu().numpy()


def _check(mats, b, x):
    """The forward-error bound of a backward-stable solver, n eps cond."""
    for k, (A, bi, xi) in enumerate(zip(mats, b, x)):
        ref = np.linalg.solve(A, bi)
        err = np.linalg.norm(xi - ref) / np.linalg.norm(ref)
        assert err <= 4 * len(A) * EPS * np.linalg.cond(A), (k, err)


def test_one_by_one_systems(cuda_lib):
    """512 systems [[1]] and [[1j]] in turn: only the even ones are looked at for the phases."""
    mats = [np.array([[1.0 + 0j]]) if k % 2 == 0 else np.array([[1j]]) for k in range(512)]
    b = np.full((512, 1), 1.0 + 2.0j)
    _check(mats, b, _solve(mats, 0, b))


@pytest.mark.parametrize("n,r", [(6, 0), (24, 2)])
@pytest.mark.parametrize("phases", [False, True])
@pytest.mark.parametrize("other", ["system", "row", "first row", "column", "border", "entries", "none"])
def test_a_system_outside_the_sample(other, phases, n, r, rng, cuda_lib):
    batch = 520
    mats = _mats(rng, batch, n, r, phases)
    A = mats[7]
    if other == "system":
        A *= 1j
    elif other == "row":
        A[n - 2] *= 1j
    elif other == "first row":
        A[r] *= -1j
    elif other == "column":
        A[:, n - 1] *= 1j
    elif other == "border":
        A[0] *= 1j
    elif other == "entries":
        A *= np.exp(1j * rng.uniform(0, 6, (n, n)))
    b = rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))
    _check(mats, b, _solve(mats, r, b))
