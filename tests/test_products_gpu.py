"""GPU: the monomials of F, with coefficients of +-1 and up to two factors alone (no product beside the
fused multiply-add) and with others among them, against the oracle's F. At 16 modes per direction the
grids are the oracle's, so that cubic and quartic terms alias alike."""
from __future__ import annotations

import copy

import numpy as np
import pytest

from _step_cases import template

pytestmark = pytest.mark.gpu

SIMPLE = [(-1.0, (0, 1)), (1.0, (2, 3)), (-1.0, (4,)), (1.0, (5,))]


@pytest.mark.parametrize("more", [[], [(2.5, (0, 3))], [(-0.5, (1,))], [(-1.0, (0, 1, 3))], [(1.0, (2, 0, 3, 1))]])
# FP64: the bound of the other comparisons with the oracle. FP32: four products and some 20 additions of
# transforms and derivatives at 6e-8 each, on values up to 2^3 times the result's norm
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 1e-5)])
def test_F_matches_oracle(more, precision, tol, rng, cuda_lib):
    from conatus_gb300.ivp import DeviceProblem
    from oracle.ivp import OracleProblem
    tpl = copy.copy(template("rb_nz16"))
    tpl.outputs = [(e, c, SIMPLE + more) for e, c, _ in tpl.outputs]
    P = tpl.instantiate([16], None, None)
    C = []
    for b, n in zip(tpl.buckets, P.nsys):
        z = rng.standard_normal((n, b.n)) + (0 if b.kind == "real" else 1j) * rng.standard_normal((n, b.n))
        C.append((z * (1.0 + np.maximum(b.col[:, 2], 0)) ** -2.5).astype(np.complex128))
    dev = DeviceProblem(P, precision)
    dev.autotune = False
    out = dev.zeros()
    dev.F(dev.to_device(C), out)
    for got, want in zip(dev.to_host(out), OracleProblem(P).F(C)):
        assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)
