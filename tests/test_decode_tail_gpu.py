"""Decode attention: cache rows past the end hold NaN and infinities, and lengths end at every kind of place inside a tile."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("length", [1, 15, 16, 63, 64, 65, 127, 128, 129, 200, 700])
@pytest.mark.parametrize("batch,heads", [(1, 2), (40, 8)])
def test_rows_past_the_end(hd, length, batch, heads):
    g = torch.Generator(device="cuda").manual_seed(length)
    S = 704
    k, v = (torch.randn(batch, heads, S, hd, device="cuda", generator=g).bfloat16() for _ in range(2))
    k[:, :, length:], v[:, :, length:] = float("nan"), float("inf")
    q = torch.randn(batch, heads * hd, device="cuda", generator=g).bfloat16()
    out = K.decode_attn(q, k, v, length).double().reshape(batch, heads, hd)
    s = torch.einsum("bhd,bhsd->bhs", q.double().reshape(batch, heads, hd), k[:, :, :length].double()) / hd ** 0.5
    ref = torch.einsum("bhs,bhsd->bhd", torch.softmax(s, -1), v[:, :, :length].double())
    # fp32 throughout and one rounding to bf16: at most 2^-9 in the norm
    assert float((out - ref).norm() / ref.norm()) <= 2.0 ** -9 + 1e-6
    torch.cuda.synchronize()
    K.check_status()
