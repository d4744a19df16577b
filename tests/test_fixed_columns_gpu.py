"""GPU: the fixed-point transforms with several columns to a block (2, 4 and 8, by the number of columns;
16 by the right-hand side's tuning), ragged last blocks and odd last pairs, columns held in registers and
read again: a column's result does not depend on its neighbours (the bits of the same column alone), and is
that of an extended-precision transform."""
from __future__ import annotations

import numpy as np
import pytest

from _step_cases import template
from test_fixed_transforms_gpu import dft, run, tol

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# at least 304 blocks (two an SM) of 2, 4 and 8 columns, never whole blocks
SHAPES = [(1, 613), (3, 437), (5, 499)]
LENGTHS = [75, 96, 288, 375, 500]                # 8 columns of 75 and 96 stay in registers, the others not


def _columns(rng, shape):
    """Columns over many orders of magnitude, some zero."""
    x = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    x = x * 10.0 ** rng.integers(-60, 60, (shape[0], 1, shape[2]))
    return x * (rng.random((shape[0], 1, shape[2])) > 0.05)


def _sample(rng, inner):
    """Columns at the ends of the blocks of 2, 4 and 8, the last ones, and some between."""
    return sorted({0, 1, 2, 3, 4, 7, 8, 9, 15, 16, inner - 1, inner - 2, inner - 3, inner // 2, *rng.integers(0, inner, 6).tolist()})


def _close(got, re, im, L, norm):
    err = np.sqrt(np.sum((got.real - re) ** 2 + (got.imag - im) ** 2, axis=0))
    assert np.all(err <= tol(L) * norm), float(np.max(err / np.maximum(norm, 1e-300)))


@pytest.mark.parametrize("L", LENGTHS)
@pytest.mark.parametrize("outer,inner", SHAPES)
def test_complex_axis(outer, inner, L):
    rng = np.random.default_rng(L + outer)
    nc = 2 * ((2 * L // 3 + 1) // 2)
    K = nc // 2
    keep = [k if k < K else L - (nc - k) for k in range(nc)]
    x = _columns(rng, (outer, L, inner))
    y = run("cng_fft_axis", 1, x, (outer, nc, inner), torch.complex128, outer, inner, nc, L)
    c = _columns(rng, (outer, nc, inner))
    z = run("cng_fft_axis", 0, c, (outer, L, inner), torch.complex128, outer, inner, nc, L)
    for o in range(outer):
        cols = _sample(rng, inner)
        for k in cols:
            assert np.array_equal(y[o, :, k], run("cng_fft_axis", 1, x[o, :, k:k + 1], (nc, 1), torch.complex128, 1, 1, nc, L)[:, 0])
            assert np.array_equal(z[o, :, k], run("cng_fft_axis", 0, c[o, :, k:k + 1], (L, 1), torch.complex128, 1, 1, nc, L)[:, 0])
    re, im = dft(x[-1][:, cols], -1, L)
    norm = np.sqrt(np.sum(np.abs(x[-1][:, cols]).astype(np.longdouble) ** 2, axis=0) / L)
    rows = [k for k in range(nc) if k != K]
    _close(y[-1][rows][:, cols], re[keep][rows] / L, im[keep][rows] / L, L, norm)
    full = np.zeros((L, len(cols)), complex)
    full[keep] = c[-1][:, cols]
    full[keep[K]] = 0
    re, im = dft(full, +1, L)
    _close(z[-1][:, cols], re, im, L, np.sqrt(np.sum(re ** 2 + im ** 2, axis=0)))


@pytest.mark.parametrize("L", LENGTHS)
@pytest.mark.parametrize("outer,inner", [(1, 1225), (3, 873), (5, 997), (2, 2490)])
def test_real_axis(outer, inner, L):
    """Pairs of adjacent columns, the last one alone where their number is odd."""
    rng = np.random.default_rng(L + inner)
    K = L // 3
    g = _columns(rng, (outer, L, inner)).real
    g[..., 1::2] = g[..., 0:inner - inner % 2:2][:, ::-1] * 0.7       # a pair's columns share a scale
    y = run("cng_rfft_axis", 1, g, (outer, K, inner), torch.complex128, outer, inner, K, L)
    c = _columns(rng, (outer, K, inner))
    c[:, 0] = c[:, 0].real
    c[..., 1::2] = c[..., 0:inner - inner % 2:2] * 0.7
    z = run("cng_rfft_axis", 0, c, (outer, L, inner), torch.float64, outer, inner, K, L)
    for o in range(outer):
        pairs = sorted({k // 2 * 2 for k in _sample(rng, inner)})
        for k in pairs:
            w = min(2, inner - k)
            assert np.array_equal(y[o, :, k:k + w], run("cng_rfft_axis", 1, g[o, :, k:k + w], (K, w), torch.complex128, 1, w, K, L))
            assert np.array_equal(z[o, :, k:k + w], run("cng_rfft_axis", 0, c[o, :, k:k + w], (L, w), torch.float64, 1, w, K, L))
    cols = pairs
    re, im = dft(g[-1][:, cols].astype(complex), -1, L)
    _close(y[-1][:, cols], re[:K] / L, im[:K] / L, L, 1.5 * np.sqrt(np.sum(g[-1][:, cols].astype(np.longdouble) ** 2, axis=0) / L))
    full = np.zeros((L, len(cols)), complex)
    full[:K] = c[-1][:, cols]
    full[L - K + 1:] = c[-1][:, cols][1:][::-1].conj()
    re, _ = dft(full, +1, L)
    _close(z[-1][:, cols], re, 0.0, L, 1.5 * np.sqrt(np.sum(re ** 2, axis=0)))


@pytest.mark.parametrize("M,N", [(96, 64), (200, 129), (288, 192), (500, 333)])
@pytest.mark.parametrize("ncols", [613, 1311, 2495])
def test_chebyshev(M, N, ncols):
    rng = np.random.default_rng(M + ncols)
    c = _columns(rng, (1, N, ncols))[0].T.copy()
    f = run("cng_cheb_transform", 0, c, (ncols, M), torch.complex128, ncols, N, M)
    g = _columns(rng, (1, M, ncols))[0].T.copy()
    y = run("cng_cheb_transform", 1, g, (ncols, N), torch.complex128, ncols, N, M)
    cols = _sample(rng, ncols)
    for k in cols:
        assert np.array_equal(f[k], run("cng_cheb_transform", 0, c[k:k + 1], (1, M), torch.complex128, 1, N, M)[0])
        assert np.array_equal(y[k], run("cng_cheb_transform", 1, g[k:k + 1], (1, N), torch.complex128, 1, N, M)[0])
    pi = np.arctan2(np.longdouble(0), np.longdouble(-1))
    ang = (np.outer(2 * np.arange(M) + 1, np.arange(M)) % (4 * M)).astype(np.longdouble) * pi / (2 * M)
    T = np.cos(ang) * np.where(np.arange(M) % 2, -1, 1)
    cs, gs = c[cols].T, g[cols].T
    re, im = T[:, :N] @ cs.real.astype(np.longdouble), T[:, :N] @ cs.imag.astype(np.longdouble)
    _close(f[cols].T, re, im, M, 2 * np.sqrt(np.sum(re ** 2 + im ** 2, axis=0)))
    W = T.T[:N] * 2 / M
    W[0] /= 2
    re, im = W @ gs.real.astype(np.longdouble), W @ gs.imag.astype(np.longdouble)
    _close(y[cols].T, re, im, M, 2 * np.sqrt(2 * np.sum(np.abs(gs).astype(np.longdouble) ** 2, axis=0) / M))


@pytest.mark.parametrize("tname,sizes", [("rb_nz16", [48]), ("channel_ny17", [14, 6])])
def test_columns_and_threads_of_a_block_do_not_change_a_bit(tname, sizes, rng, cuda_lib):
    """The right-hand side by columns per block (1 to 32) and threads."""
    from conatus_gb300 import autotune
    from conatus_gb300.ivp import DeviceProblem
    dev = DeviceProblem(template(tname).instantiate(sizes), "fp64")
    x = dev.zeros()
    x.copy_(torch.as_tensor(rng.standard_normal(dev.n_total) + 1j * rng.standard_normal(dev.n_total)))
    ref = None
    for q, t in ((0, 0), (1, 64), (2, 96), (3, 128), (4, 256), (8, 64), (16, 256), (32, 512)):
        autotune._set_rhs_tuning(dev, q, t)
        out = dev.zeros()
        dev.F(x, out)
        torch.cuda.synchronize()
        ref = out if ref is None else ref
        assert torch.equal(out, ref), (q, t)
