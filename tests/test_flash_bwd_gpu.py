"""The two backward kernels of attention at both head dims: less than a tile, edges of tiles, one to several tiles per item and items per
CTA, full and causal, gradients into the columns of one packed row, queries scaled so that probabilities are far from uniform."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("batch,seq,heads", [(1, 1, 2), (2, 65, 1), (1, 127, 3), (2, 128, 1), (1, 129, 3), (2, 300, 2), (1, 513, 1), (3, 640, 25), (149, 100, 1)])
def test_backward(hd, causal, batch, seq, heads):
    g = torch.Generator(device="cuda").manual_seed(seq + heads)
    D = heads * hd
    qkv = torch.randn(batch * seq, 3 * D, device="cuda", generator=g)
    qkv[:, :D] *= 2.0
    qkv = qkv.bfloat16()
    do = torch.randn(batch * seq, D, device="cuda", generator=g).bfloat16()
    parts = [qkv[:, i * D:(i + 1) * D] for i in range(3)]
    o, lse = K.flash_fwd(*parts, batch, seq, heads, hd, causal=causal)
    got = K.flash_bwd(*parts, o, do, lse, batch, seq, heads, hd, causal=causal)
    again = K.flash_bwd(*parts, o, do, lse, batch, seq, heads, hd, causal=causal)
    q, k, v, w = (t.double().reshape(batch, seq, heads, hd).transpose(1, 2) for t in (*parts, do))
    scale = hd ** -0.5
    s = q @ k.transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(~torch.ones(seq, seq, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    p = torch.softmax(s, -1)
    dp = w @ v.transpose(-1, -2)
    ds = p * (dp - (w * (p @ v)).sum(-1, keepdim=True)) * scale
    # Three roundings to bf16 (2^-9 each) stand between exact sums and the result: O (in delta), P or dS, the gradient.  One key leaves
    # nothing of dS but the rounding of O, which is measured against the term that cancels.
    floor = 2.0 ** -9 * float((p * dp).norm() * scale * q.norm()) if seq == 1 else 0.0
    for name, a, b, ref in zip("qkv", got, again, (ds @ k, ds.transpose(-1, -2) @ q, p.transpose(-1, -2) @ w)):
        ref = ref.transpose(1, 2).reshape(batch * seq, D)
        assert float((a.double() - ref).norm()) <= 2.0 ** -7 * float(ref.norm()) + floor, name
        assert torch.equal(a, b), name                         # one writer per element, sums in a fixed order
    torch.cuda.synchronize()
    K.check_status()
