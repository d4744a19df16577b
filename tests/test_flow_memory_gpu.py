"""GPU: the operations that a handle of host matrices builds unasked: at most 1 GB as allocated (whole
chunks of slots, not an estimate), and none where the device has no room for them; the handle is made
and solves all the same."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

GB = 1 << 30
CHUNK = 6144                        # bytes of 16 slots of 32 operations of 12 bytes


def _diagonal(rng, batch):
    """`batch` systems [[d]]: a chunk each, of which one operation is used."""
    from conatus_gb300 import core
    d = rng.uniform(0.5, 2.0, batch)
    ip, ix = np.array([0, 1], np.int32), np.array([0], np.int32)
    live = core.pool_stats()[0]
    h = core.cuda.BandedBatchD([(1, ip, ix, d[k:k + 1]) for k in range(batch)], [])
    return h, d, core.pool_stats()[0] - live


def _check(h, d):
    x = torch.ones((len(d), 1), dtype=torch.float64, device="cuda")
    h.solve_ptr(x.data_ptr(), len(d), 1)
    assert np.allclose(x.cpu().numpy()[:, 0] * d, 1.0, rtol=1e-15, atol=0)


@pytest.mark.parametrize("batch,built", [(20000, True), (GB // CHUNK - 2000, True), (GB // CHUNK + 1000, False)])
def test_at_most_a_gigabyte(batch, built, rng, cuda_lib):
    h, d, held = _diagonal(rng, batch)
    assert held < GB + batch * 64
    assert (held >= batch * CHUNK) == built
    _check(h, d)


def test_no_room(rng, cuda_lib):
    """Room for the factors (some 5 MB), not for the operations (0.9 GB)."""
    h, d, _ = _diagonal(rng, 1000)                       # every kernel loaded
    _check(h, d)
    del h
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - 500 * 2 ** 20, dtype=torch.uint8, device="cuda")
    try:
        h, d, held = _diagonal(rng, 150000)
        assert held < 64 * 2 ** 20
        _check(h, d)
    finally:
        del hold
        torch.cuda.empty_cache()
