"""fp32 attention with one and with four groups of threads to a row, at widths and lengths off the tile grid and on both sides of the rule."""
import pytest
import torch

from device_time import graph_us
from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [8, 30, 32, 48, 64])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("batch,seq,heads", [(1, 1, 1), (2, 33, 2), (1, 128, 4), (2, 257, 1), (24, 100, 4), (64, 16, 4), (75, 16, 4)])
def test_attention(hd, causal, batch, seq, heads):
    g = torch.Generator(device="cuda").manual_seed(hd + seq)
    D = heads * hd
    qkv, do = torch.randn(batch * seq, 3 * D, device="cuda", generator=g), torch.randn(batch * seq, D, device="cuda", generator=g)
    q, k, v = qkv[:, :D], qkv[:, D:2 * D], qkv[:, 2 * D:]
    o, lse = K.flash_fwd(q, k, v, batch, seq, heads, hd, causal=causal)
    got = K.flash_bwd(q, k, v, o, do, lse, batch, seq, heads, hd, causal=causal)
    leaves = [t.double().reshape(batch, seq, heads, hd).transpose(1, 2).requires_grad_(True) for t in (q, k, v)]
    ref = torch.nn.functional.scaled_dot_product_attention(*leaves, is_causal=causal).transpose(1, 2).reshape(batch * seq, D)
    grads = torch.autograd.grad(ref, leaves, do.double())
    # __expf of arguments up to 2^4 carries 2^-20; sums of 257 products
    for a, e in zip((o, *got), (ref, *[x.transpose(1, 2).reshape(batch * seq, D) for x in grads])):
        # (a gradient that cancels to nothing, as with one key, is measured against the upstream gradient)
        assert float((a.double() - e.detach()).norm() / torch.maximum(e.detach().norm(), do.double().norm())) <= 8e-6


# With a CTA or more per SM a row shared by more threads does more work per score: there a full mask took 1.5 times a causal one, where the
# form with one group of threads to a row takes the same time for both.
def test_many_rows_take_the_wide_form():
    def us(causal):
        qkv = torch.randn(8 * 512, 3 * 256, device="cuda")
        return graph_us(*[lambda: K.flash_fwd(qkv[:, :256], qkv[:, 256:512], qkv[:, 512:], 8, 512, 4, 64, causal=causal)] * 4)

    assert us(False) <= 1.25 * us(True)
