"""The two-tile forward kernel at both head dims: odd tile counts, sequences off the tile grid, full and causal, packed rows."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("batch,seq,heads", [(1, 1, 1), (1, 100, 2), (2, 128, 1), (1, 129, 3), (2, 300, 2), (1, 513, 1), (3, 640, 25), (1, 1500, 4)])
def test_forward(hd, causal, batch, seq, heads):
    g = torch.Generator(device="cuda").manual_seed(seq + heads)
    D = heads * hd
    qkv = torch.randn(batch * seq, 3 * D, device="cuda", generator=g)
    qkv[:, :D] *= 3.0                                           # rows whose maximum moves by more than the lazy threshold
    qkv = qkv.bfloat16()
    o, lse = K.flash_fwd(qkv[:, :D], qkv[:, D:2 * D], qkv[:, 2 * D:], batch, seq, heads, hd, causal=causal)
    q, k, v = (t.double().reshape(batch, seq, heads, hd).transpose(1, 2) for t in (qkv[:, :D], qkv[:, D:2 * D], qkv[:, 2 * D:]))
    s = q @ k.transpose(-1, -2) / hd ** 0.5
    if causal:
        s = s.masked_fill(~torch.ones(seq, seq, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    ref = (torch.softmax(s, -1) @ v).transpose(1, 2).reshape(batch * seq, D)
    # probabilities and output are rounded to bf16 once each (2^-9)
    assert float((o.double() - ref).norm() / ref.norm()) <= 2.0 ** -8
    assert (lse.double() - torch.logsumexp(s, -1)).abs().max().item() <= 1e-4
    torch.cuda.synchronize()
    K.check_status()
