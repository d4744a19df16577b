"""GPU: F in FP64 with Fourier directions (a block per system unpacks the state, one warp per y-group)
against the oracle's F: Chebyshev sizes around the derivative's eight segments of each parity, one and
two Fourier directions, mean modes, more systems than one block of warps."""
from __future__ import annotations

import numpy as np
import pytest

from _step_cases import template

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tname,sizes", [("rb_nz16", [8]), ("rb_nz32_ra", [20]), ("rb_nz48_ra", [34]), ("rb_nz80_ra", [16]),
                                         ("rb_nz96_ra", [64]), ("channel_ny17", [4, 4]), ("channel_ny17", [10, 14]),
                                         ("channel_ny129", [6, 8])])
def test_F_matches_oracle(tname, sizes, rng, cuda_lib):
    from conatus_gb300.ivp import DeviceProblem
    from oracle.ivp import OracleProblem
    tpl = template(tname)
    P = tpl.instantiate(sizes, None, {"Ra": 3e4} if tpl.linear_params else None)
    C = []
    for b, n in zip(tpl.buckets, P.nsys):
        z = rng.standard_normal((n, b.n)) + (0 if b.kind == "real" else 1j) * rng.standard_normal((n, b.n))
        C.append((z * (1.0 + np.maximum(b.col[:, 2], 0)) ** -1.5).astype(np.complex128))
    dev = DeviceProblem(P, "fp64")
    dev.autotune = False
    out = dev.zeros()
    dev.F(dev.to_device(C), out)
    # the bound of the other comparisons of F with the oracle
    for got, want in zip(dev.to_host(out), OracleProblem(P).F(C)):
        assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
