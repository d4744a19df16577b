"""The fixed-point FP64 transforms against extended-precision DFTs: every radix, prime-power block and
rescaled length, ragged batches, both directions; columns of very different sizes, zeros, denormals,
the largest exponents and non-finite entries side by side."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps
LENGTHS = [1, 2, 3, 4, 5, 8, 9, 15, 16, 18, 25, 27, 32, 45, 48, 75, 96, 125, 128, 135, 200, 243, 256, 288,
           300, 320, 375, 384, 500, 512, 768, 1000]


def tol(L):
    """The FP64 transforms' error, relative L2 per column: a rounding per halving of the length (and one
    for the final rounding)."""
    return EPS * (1 + 0.5 * np.log2(L + 1))


def dft(x, sign, L):
    """Extended-precision DFT along axis 0 (the angles reduced exactly)."""
    n = np.arange(L)
    ang = (np.outer(n, n) % L).astype(np.longdouble) * (2 * np.arctan2(np.longdouble(0), np.longdouble(-1))) / L
    c, s = np.cos(ang), sign * np.sin(ang)
    re, im = x.real.astype(np.longdouble), x.imag.astype(np.longdouble)
    return c @ re - s @ im, s @ re + c @ im


def check(got, re, im, L, what):
    err = np.sqrt(np.sum((got.real - re) ** 2 + (got.imag - im) ** 2, axis=0))
    ref = np.sqrt(np.sum(re ** 2 + im ** 2, axis=0))
    assert np.all(err <= tol(L) * ref), (what, L, float(np.max(err / ref)) / EPS)


def run(name, fwd, x, shape, dtype, *sizes):
    from conatus_gb300 import _lib
    a = torch.as_tensor(np.ascontiguousarray(x), device="cuda")
    out = torch.full(shape, 7.0, dtype=dtype, device="cuda")
    _lib.call(name, fwd, a.data_ptr(), out.data_ptr(), *sizes, torch.cuda.current_stream().cuda_stream)
    return out.cpu().numpy()


def columns(rng, L, inner):
    """Columns of flat and of decaying magnitude, over 200 orders of magnitude."""
    x = rng.standard_normal((L, inner)) + 1j * rng.standard_normal((L, inner))
    x[:, ::2] *= (1.0 + np.arange(L))[:, None] ** -1.5
    return x * 10.0 ** rng.integers(-100, 100, inner)


@pytest.mark.parametrize("L", LENGTHS)
@pytest.mark.parametrize("inner", [1, 13])
def test_complex_axis(L, inner):
    rng = np.random.default_rng(L)
    nc = 2 * ((2 * L // 3 + 1) // 2)
    if nc > L:
        nc -= 2
    K = nc // 2
    x = columns(rng, L, inner)
    y = run("cng_fft_axis", 1, x, (nc, inner), torch.complex128, 1, inner, nc, L) if nc else None
    if nc:
        re, im = dft(x, -1, L)
        keep = [k if k < K else L - (nc - k) for k in range(nc)]
        re, im = re[keep] / L, im[keep] / L
        err = np.sqrt(np.sum(np.delete((y.real - re) ** 2 + (y.imag - im) ** 2, K, 0), axis=0))
        norm = np.sqrt(np.sum(np.abs(x).astype(np.longdouble) ** 2, axis=0) / L)
        assert np.all(err <= tol(L) * norm) and np.all(y[K] == 0)
    c = columns(rng, max(nc, 1), inner)[:nc]
    z = run("cng_fft_axis", 0, c, (L, inner), torch.complex128, 1, inner, nc, L) if nc else None
    if nc:
        full = np.zeros((L, inner), np.complex128)
        for k in range(nc):
            if k != K:
                full[k if k < K else L - (nc - k)] = c[k]
        if np.any(full):
            check(z, *dft(full, +1, L), L, "backward")


@pytest.mark.parametrize("L", LENGTHS)
@pytest.mark.parametrize("inner", [2, 7])
def test_real_axis(L, inner):
    rng = np.random.default_rng(L + 1)
    K = max(1, min(L // 3, (L + 1) // 2))
    g = columns(rng, L, inner).real
    # the two columns of a pair share one scale: keep them within what the bound is stated for
    g[:, 1::2] = g[:, 0:inner - inner % 2:2][::-1] * 0.7
    y = run("cng_rfft_axis", 1, g, (K, inner), torch.complex128, 1, inner, K, L)
    re, im = dft(g.astype(np.complex128), -1, L)
    err = np.sqrt(np.sum((y.real - re[:K] / L) ** 2 + (y.imag - im[:K] / L) ** 2, axis=0))
    assert np.all(err <= 1.5 * tol(L) * np.sqrt(np.sum(g.astype(np.longdouble) ** 2, axis=0) / L))
    c = columns(rng, K, inner)
    c[0] = c[0].real
    c[:, 1::2] = c[:, 0:inner - inner % 2:2] * 0.7
    z = run("cng_rfft_axis", 0, c, (L, inner), torch.float64, 1, inner, K, L)
    full = np.zeros((L, inner), np.complex128)
    full[:K] = c
    for k in range(1, K):
        full[L - k] = c[k].conj()
    re, _ = dft(full, +1, L)
    err = np.sqrt(np.sum((z - re) ** 2, axis=0))
    assert np.all(err <= 1.5 * tol(L) * np.sqrt(np.sum(re ** 2, axis=0)))


@pytest.mark.parametrize("M,N", [(2, 1), (2, 2), (4, 3), (6, 5), (18, 12), (30, 30), (32, 21), (96, 64), (200, 129),
                                 (250, 166), (256, 256), (384, 256), (400, 257), (768, 512)])
@pytest.mark.parametrize("ncols", [1, 11])
def test_chebyshev(M, N, ncols):
    rng = np.random.default_rng(M + N)
    c = columns(rng, N, ncols).T
    f = run("cng_cheb_transform", 0, c, (ncols, M), torch.complex128, ncols, N, M)
    pi = np.arctan2(np.longdouble(0), np.longdouble(-1))
    # T_k(-cos(pi (j + 1/2) / M)) = (-1)^k cos(pi k (2j + 1) / 2M)
    ang = (np.outer(2 * np.arange(M) + 1, np.arange(M)) % (4 * M)).astype(np.longdouble) * pi / (2 * M)
    T = np.cos(ang) * np.where(np.arange(M) % 2, -1, 1)
    re, im = T[:, :N] @ c.real.T.astype(np.longdouble), T[:, :N] @ c.imag.T.astype(np.longdouble)
    err = np.sqrt(np.sum((f.T.real - re) ** 2 + (f.T.imag - im) ** 2, axis=0))
    assert np.all(err <= 2 * tol(M) * np.sqrt(np.sum(re ** 2 + im ** 2, axis=0)))
    g = columns(rng, M, ncols).T
    y = run("cng_cheb_transform", 1, g, (ncols, N), torch.complex128, ncols, N, M)
    W = T.T[:N] * 2 / M
    W[0] /= 2
    re, im = W @ g.real.T.astype(np.longdouble), W @ g.imag.T.astype(np.longdouble)
    err = np.sqrt(np.sum((y.T.real - re) ** 2 + (y.T.imag - im) ** 2, axis=0))
    norm = np.sqrt(2 * np.sum(np.abs(g.T).astype(np.longdouble) ** 2, axis=0) / M)
    assert np.all(err <= 2 * tol(M) * norm)


@pytest.mark.parametrize("L", [24, 288, 512])
def test_extreme_columns(L):
    """A zero column, one of denormals, one at the top of the range, NaN and infinity, and an ordinary
    column between them that none of these may touch."""
    rng = np.random.default_rng(5)
    x = rng.standard_normal((L, 6)) + 1j * rng.standard_normal((L, 6))
    x[:, 0] = 0.0
    x[:, 1] *= 1e-310
    x[:, 2] *= 1e304
    x[3, 3] = np.nan
    x[5, 4] = np.inf
    y = run("cng_fft_axis", 0, x, (L, 6), torch.complex128, 1, 6, L, L)
    x[L // 2] = 0.0
    assert np.all(y[:, 0] == 0)
    re, im = dft(x[:, [2, 5]], +1, L)
    check(y[:, [2, 5]], re, im, L, "extreme")
    re, im = dft(x[:, [1]], +1, L)
    assert np.max(np.abs(y[:, 1].real - re[:, 0])) <= 1e-322 + 4 * EPS * np.max(np.abs(re))
    assert not np.isfinite(y[:, 3:5]).any()
    z = run("cng_fft_axis", 0, x * 2.0 ** 300, (L, 6), torch.complex128, 1, 6, L, L)
    assert np.array_equal(z[:, 5], y[:, 5] * 2.0 ** 300)       # a power of two changes no rounding
