"""RoPE with the heads of a row dealt to threads, against a 64-bit statement."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


def _rel(a, e):
    return float((a.double().cpu() - e.double().cpu()).norm() / e.double().norm().cpu().clamp_min(1e-30))


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("rows,heads,seq", [(1, 1, 1), (3, 7, 1), (32, 64, 1), (40, 10, 8), (6000, 6, 3000)])
def test_rope_head_groups(hd, rows, heads, seq):
    g = torch.Generator(device="cuda").manual_seed(rows + heads)
    x = torch.randn(rows, heads * hd + 8, device="cuda", generator=g).bfloat16()
    pos = torch.full((1,), 5, dtype=torch.int32, device="cuda")
    for back in (False, True):
        got = K.rope_(x.clone(), heads, hd, seq, pos_offset=2, backward=back, pos_dev=pos)
        ref = K.rope_(x.cpu().double(), heads, hd, seq, pos_offset=7, backward=back)
        assert torch.equal(got[:, heads * hd:], x[:, heads * hd:])
        # angles up to 3007 in fp32 (2^-24 of them) and one rounding to bf16
        assert _rel(got[:, :heads * hd], ref[:, :heads * hd]) <= 2.0 ** -8


def test_no_heads_and_no_rows():
    x = torch.randn(4, 64, device="cuda").bfloat16()
    assert torch.equal(K.rope_(x.clone(), 0, 64, 1), x)
    assert K.rope_(x[:0].clone(), 1, 64, 1).shape == (0, 64)
