"""GPU: the real transforms on reals that start 8 bytes off a 16-byte boundary (a slice of a buffer): the
results of aligned ones, bit for bit, and nothing written beside them."""
from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("outer,inner,K,L", [(1, 2, 3, 6), (2, 8, 4, 12), (3, 640, 32, 96), (2, 7, 5, 15)])
@pytest.mark.parametrize("off", [0, 1])
def test_real_axis_of_a_slice(outer, inner, K, L, off, rng, cuda_lib):
    from conatus_gb300._lib import call
    c = torch.as_tensor(rng.standard_normal((outer, K, inner)) + 1j * rng.standard_normal((outer, K, inner)), device="cuda")
    count = outer * L * inner
    ref = torch.empty(count, dtype=torch.float64, device="cuda")
    call("cng_rfft_axis", 0, c.data_ptr(), ref.data_ptr(), outer, inner, K, L, None)
    buf = torch.full((count + 2,), 7.0, dtype=torch.float64, device="cuda")
    call("cng_rfft_axis", 0, c.data_ptr(), buf[off:].data_ptr(), outer, inner, K, L, None)
    torch.cuda.synchronize()
    assert torch.equal(buf[off:off + count], ref)
    assert torch.all(buf[:off] == 7.0) and torch.all(buf[off + count:] == 7.0)
    back, back2 = torch.empty_like(c), torch.empty_like(c)
    call("cng_rfft_axis", 1, ref.data_ptr(), back.data_ptr(), outer, inner, K, L, None)
    call("cng_rfft_axis", 1, buf[off:].data_ptr(), back2.data_ptr(), outer, inner, K, L, None)
    torch.cuda.synchronize()
    assert torch.equal(back, back2)
