"""Attention backward where a CTA works through several items of different lengths: its barriers go on from one to the next, and an item's last
tile gives no turn to the issuer of dK and dP."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("batch,seq", [(240, 100), (120, 129), (100, 384), (60, 641)])     # one, two, three and six tiles, 480 to 720 items
def test_items_in_a_row(hd, causal, batch, seq):
    heads = 2
    D = heads * hd
    g = torch.Generator(device="cuda").manual_seed(seq + hd)
    qkv = torch.randn(batch * seq, 3 * D, device="cuda", generator=g).bfloat16()
    do = torch.randn(batch * seq, D, device="cuda", generator=g).bfloat16()
    parts = [qkv[:, i * D:(i + 1) * D] for i in range(3)]
    o, lse = K.flash_fwd(*parts, batch, seq, heads, hd, causal=causal)
    got = [t.clone() for t in K.flash_bwd(*parts, o, do, lse, batch, seq, heads, hd, causal=causal)[:3]]
    again = K.flash_bwd(*parts, o, do, lse, batch, seq, heads, hd, causal=causal)[:3]
    assert all(torch.equal(a, b) for a, b in zip(got, again))                            # one writer per element, the same order every time
    mask = torch.ones(seq, seq, dtype=torch.bool, device="cuda").triu(1)
    for b0 in range(0, batch, 20):                                                       # in 64 bits, some sequences at a time
        rows = slice(b0 * seq, (b0 + 20) * seq)
        x = qkv[rows].double().requires_grad_(True)
        q, k, v = (x[:, i * D:(i + 1) * D].reshape(20, seq, heads, hd).transpose(1, 2) for i in range(3))
        s = q @ k.transpose(-1, -2) / hd ** 0.5
        if causal:
            s = s.masked_fill(mask, float("-inf"))
        ref, = torch.autograd.grad((torch.softmax(s, -1) @ v).transpose(1, 2).reshape(20 * seq, D), x, do[rows].double())
        for i in range(3):
            r = ref[:, i * D:(i + 1) * D]
            # probabilities, their gradients, the output of the forward pass and the results are rounded to bf16: in the norm up to 2^-9 each
            assert float((got[i][rows].double() - r).norm()) <= 2.0 ** -7 * float(r.norm())
    torch.cuda.synchronize()
    K.check_status()
