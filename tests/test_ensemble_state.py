"""CPU: FourierEnsemble.set_state takes its members' states as any iterable of anything that ravels to
complex numbers."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

def _forms(C):
    return {
        "list": list(C),
        "tuple": tuple(C),
        "generator": (c for c in C),
        "map": map(np.copy, C),
        "rows": [c[None] for c in C],
        "columns": [c[:, None] for c in C],
        "mixed ranks": [c if k % 2 else c[None] for k, c in enumerate(C)],
        "lists": [c.tolist() for c in C],
        "strided": [np.repeat(c, 2)[::2] for c in C],
        "one list among arrays": [C[0].tolist()] + list(C[1:]),
        "object": [c.astype(object) for c in C],
        "complex64 of the same": [c.astype(np.complex64) for c in C],
        "tensors": [torch.as_tensor(c) for c in C],
    }


@pytest.fixture
def e(monkeypatch):
    """The state of an ensemble of members of 8, 12 and 8 amplitudes, on the host."""
    from conatus_gb300 import ensemble
    monkeypatch.setattr(ensemble, "_torch", lambda: torch)
    e = ensemble.FourierEnsemble.__new__(ensemble.FourierEnsemble)
    e.n_total, e.order = 28, 2
    e.X = torch.zeros(28, dtype=torch.complex128)
    return e


@pytest.mark.parametrize("form", list(_forms([np.zeros(1, complex)])))
def test_members_in_every_form(form, e, rng):
    C = [(rng.integers(-9, 10, k) + 1j * rng.integers(-9, 10, k)).astype(complex) for k in (8, 12, 8)]
    e.set_state(_forms(C)[form])
    assert np.array_equal(e.X.cpu().numpy(), np.concatenate(C))


def test_single_numbers(e):
    """Members of one amplitude as 0-d arrays beside the other's vector."""
    parts = [np.array(1.0 + 0j)] * 8 + [np.arange(20) * (1 + 1j)]
    e.set_state(parts)
    assert np.array_equal(e.X.cpu().numpy(), np.concatenate([np.ravel(p) for p in parts]))


def test_wrong_sizes_are_refused(e):
    with pytest.raises(ValueError):
        e.set_state([np.zeros(8, complex), np.zeros(8, complex)])
    with pytest.raises(ValueError):
        e.set_state([])
