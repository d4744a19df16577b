"""GPU: the scheduled solve (flow_solve.cu): bands, border rows and sizes at their edges, real systems and
complex ones that are real up to powers of i, every way a right-hand side comes in; what it does not
take stays with the band kernel; the column sweeps' bits, FP64 and FP32, whole and by system ranges,
shared pairs included."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

from _step_cases import template

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def systems(rng, batch, n, kl, ku, r, complex_):
    """Random bordered banded systems (pivoting among them), border rows first, in the real form: entry
    (k, j) carries i^(p_k - q_j)."""
    p, q = rng.integers(0, 2, n), rng.integers(0, 2, n)
    p[:r] = q[:r]
    out = []
    for _ in range(batch):
        A = np.zeros((n, n))
        for d in range(-min(kl, n - 1), min(ku, n - 1) + 1):
            A += np.diag(rng.standard_normal(n - abs(d)), d)
        A += 2.0 * np.eye(n)
        A[:r] = rng.standard_normal((r, n))
        A[np.arange(r), np.arange(r)] += 4.0
        if complex_:
            A = A * np.where(p[:, None] == q[None], 1, np.where(p[:, None] > q[None], 1j, -1j))
        out.append(A)
    return out


def handle(mats, r):
    from conatus_gb300 import core
    cls = core.cuda.BandedBatchZ if np.iscomplexobj(mats[0]) else core.cuda.BandedBatchD
    csr = [sp.csr_matrix(A) for A in mats]
    return cls([(A.shape[0], C.indptr, C.indices, C.data) for A, C in zip(mats, csr)], list(range(r)))


def rhs(rng, batch, n, complex_):
    b = rng.standard_normal((batch, n))
    return b + 1j * rng.standard_normal((batch, n)) if complex_ else b


def check(mats, b, x):
    """The forward-error bound of a backward-stable solver, n eps cond."""
    for A, bi, xi in zip(mats, b, x):
        ref = np.linalg.solve(A, bi)
        assert np.linalg.norm(xi - ref) <= 4 * len(A) * EPS * np.linalg.cond(A) * np.linalg.norm(ref)


@pytest.mark.parametrize("complex_", [False, True])
@pytest.mark.parametrize("n,kl,ku,r", [(1, 0, 0, 0), (2, 1, 0, 1), (3, 0, 2, 3), (15, 2, 3, 0), (31, 4, 20, 3), (32, 0, 5, 0),
                                       (33, 5, 0, 2), (40, 33, 3, 1), (64, 1, 1, 1), (70, 40, 38, 2), (100, 7, 40, 12),
                                       (131, 2, 2, 33)])
def test_matches_dense(n, kl, ku, r, complex_, rng, cuda_lib):
    mats = systems(rng, 3, n, kl, ku, r, complex_)
    b = rhs(rng, 3, n, complex_)
    h = handle(mats, r)
    t = torch.as_tensor(b, device="cuda")
    x = torch.empty_like(t)
    h.solve_mapped_ptr(t.data_ptr(), 0, x.data_ptr(), 0)
    check(mats, b, x.cpu().numpy())
    h.solve_ptr(t.data_ptr(), 3, n)                          # in place: the same operations
    assert torch.equal(t, x)


def test_maps_and_split(rng, cuda_lib):
    n, r, batch = 50, 2, 4
    mats = systems(rng, batch, n, 5, 7, r, True)
    b = rhs(rng, batch, n, True)
    h = handle(mats, r)
    t = torch.as_tensor(b, device="cuda")
    x = torch.empty_like(t)
    h.solve_mapped_ptr(t.data_ptr(), 0, x.data_ptr(), 0)
    rows, cols = rng.permutation(batch * n), rng.permutation(batch * n)
    src = torch.empty(batch * n, dtype=torch.complex128, device="cuda")
    out = torch.empty_like(src)
    ri, ci = (torch.as_tensor(v, device="cuda") for v in (rows, cols))
    src[ri] = t.reshape(-1)
    h.solve_mapped_ptr(src.data_ptr(), ri.data_ptr(), out.data_ptr(), ci.data_ptr())
    assert torch.equal(out[ci], x.reshape(-1))
    both = rng.permutation(2 * batch * n)
    c, s = (torch.as_tensor(v, device="cuda") for v in (both[:batch * n].copy(), both[batch * n:].copy()))
    re = torch.empty(2 * batch * n, dtype=torch.float64, device="cuda")
    re[c], re[s] = t.reshape(-1).real, t.reshape(-1).imag
    xs = torch.empty_like(re)
    h.solve_split_ptr(re.data_ptr(), c.data_ptr(), s.data_ptr(), xs.data_ptr(), c.data_ptr(), s.data_ptr())
    assert torch.equal(torch.complex(xs[c], xs[s]), x.reshape(-1))


def test_border_rows_anywhere(rng, cuda_lib):
    from conatus_gb300 import core
    n, order = 45, None
    mats = systems(rng, 2, n, 3, 4, 3, True)
    order = [7, 30, 44] + [i for i in range(n) if i not in (7, 30, 44)]
    full = []
    for A in mats:
        B = np.empty_like(A)
        B[order] = A
        full.append(B)
    csr = [sp.csr_matrix(B) for B in full]
    h = core.cuda.BandedBatchZ([(n, C.indptr, C.indices, C.data) for C in csr], order[:3])
    b = rhs(rng, 2, n, True)
    t = torch.as_tensor(b, device="cuda")
    h.solve_ptr(t.data_ptr(), 2, n)
    check(full, b, t.cpu().numpy())


def test_other_complex_systems_keep_the_band_kernel(rng, cuda_lib):
    """One system whose entries are not real up to the phases: the batch is solved all the same."""
    n, r = 40, 2
    mats = systems(rng, 3, n, 3, 4, r, True)
    mats[2] = mats[2] * np.exp(1j * rng.uniform(0, 6, (n, n)))
    b = rhs(rng, 3, n, True)
    t = torch.as_tensor(b, device="cuda")
    handle(mats, r).solve_ptr(t.data_ptr(), 3, n)
    check(mats, b, t.cpu().numpy())


def test_a_bad_system_stays_alone(rng, cuda_lib):
    n, r = 70, 2
    mats = systems(rng, 3, n, 6, 6, r, True)
    b = rhs(rng, 3, n, True)
    h = handle(mats, r)
    ref = torch.as_tensor(b, device="cuda")
    h.solve_ptr(ref.data_ptr(), 3, n)
    b[1, 30] = np.nan
    t = torch.as_tensor(b, device="cuda")
    h.solve_ptr(t.data_ptr(), 3, n)
    assert torch.equal(t[0], ref[0]) and torch.equal(t[2], ref[2]) and torch.isnan(t[1]).any()


@pytest.mark.parametrize("tname,sizes,share", [("rb_nz16", [32], True), ("burgers_n128", None, True), ("channel_ny17", [8, 8], False),
                                               ("channel_ny17", [14, 6], True)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_the_column_sweeps_bits(tname, sizes, share, precision, rng, cuda_lib):
    """A step's buckets in one launch: the results of schedule 0 and of the split-lane schedules, bit for
    bit, whole and by system ranges."""
    from conatus_gb300 import autotune
    from conatus_gb300.ivp import DeviceProblem, _Partner
    dev = DeviceProblem(template(tname).instantiate(sizes), precision, share=share)
    dev.autotune = False
    fs = dev.factor(1.5e3, 1.0)
    fp32 = int(precision == "fp32")
    b = dev.zeros()
    b.copy_(torch.as_tensor(rng.standard_normal(dev.n_total) + 1j * rng.standard_normal(dev.n_total)))

    def solve(sched, group):
        autotune.apply(fs, sched)
        x = dev.zeros()
        for g in group:
            dev._batch_call(fs, g, b, x, None, fp32, 0, None)
        torch.cuda.synchronize()
        return x
    whole = [list(range(len(fs)))]
    like32, like16 = autotune.scheduled_schedules()
    ref = solve(0, whole)
    assert torch.equal(solve(like16, whole), ref)
    parts = []
    for k, f in enumerate(fs):
        if not isinstance(f, _Partner):
            cut = min(dev.nsys[k], 2 * ((dev.nsys[k] + 3) // 4))
            parts += [[(k, s0, s1)] for s0, s1 in ((0, cut), (cut, dev.nsys[k])) if s1 > s0]
    assert torch.equal(solve(like16, parts), ref)
    if not dev.shared:
        split = min(autotune.split_schedules())
        assert torch.equal(solve(like32, whole), solve(split, whole))
