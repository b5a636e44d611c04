"""The two-tile forward kernel at both head dims and the single-tile one at head dim 128: odd tile counts, sequences off the tile grid,
full and causal, packed rows, both sides of the line between them."""
import pytest
import torch

from device_time import graph_us
from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("batch,seq,heads", [(1, 1, 1), (1, 100, 2), (2, 128, 1), (1, 129, 3), (2, 300, 2), (1, 513, 1), (3, 640, 25), (1, 1500, 4), (149, 100, 1),
                                             (37, 300, 4), (10, 1100, 5)])
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


# While there are fewer tiles than SMs each has one of its own: half the heads take about half the time, not the time of two tiles
# that share an SM beside idle ones.
@pytest.mark.parametrize("causal", [True, False])
def test_few_tiles_take_an_sm_each(causal):
    def us(heads, seq=1024, hd=128):
        D = heads * hd
        qkv = torch.randn(seq, 3 * D, device="cuda").bfloat16()
        call = lambda: K.flash_fwd(qkv[:, :D], qkv[:, D:2 * D], qkv[:, 2 * D:], 1, seq, heads, hd, causal=causal)
        return graph_us(*[call] * 10)

    assert us(18) <= 0.75 * us(36)
