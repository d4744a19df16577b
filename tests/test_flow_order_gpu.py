"""GPU: a slot of the scheduled solve may write a row that other operations of the same slot read (x_j =
y_j / u_jj goes with the last updates by y_j): the reads come first. Systems made of such slots, with
powers of two and small whole numbers, so that every result is exact in FP64."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("n,ku,batch", [(2, 1, 1), (17, 1, 3), (33, 4, 2), (64, 7, 610), (257, 2, 5)])
def test_reads_before_writes(n, ku, batch, complex_, rng, cuda_lib):
    from conatus_gb300 import core
    # U with +-2^k on the diagonal: x whole, b = U x exact, and so is every y_j - u_ij / u_jj y_j
    U = np.zeros((n, n))
    for d in range(1, min(ku, n - 1) + 1):
        U += np.diag(rng.integers(-1, 2, n - d).astype(float), d)
    U += np.diag(2.0 ** rng.integers(0, 2, n) * rng.choice([-1, 1], n))
    C = sp.csr_matrix(U)
    kind = np.complex128 if complex_ else np.float64
    h = (core.cuda.BandedBatchZ if complex_ else core.cuda.BandedBatchD)(
        [(n, C.indptr, C.indices, C.data.astype(kind))] * batch, [])
    x = rng.integers(-8, 9, (batch, n)).astype(kind)
    if complex_:
        x = x + 1j * rng.integers(-8, 9, (batch, n))
    b = torch.as_tensor(x @ U.T.astype(kind), device="cuda")
    got = torch.empty_like(b)
    for _ in range(3):
        h.solve_mapped_ptr(b.data_ptr(), 0, got.data_ptr(), 0)
        assert torch.equal(got.cpu(), torch.as_tensor(x))
