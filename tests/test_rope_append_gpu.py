"""Rotation and cache append of one new token per sequence in one launch, against the two general kernels."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [16, 48, 64, 128])
@pytest.mark.parametrize("batch,heads,pos,offset", [(1, 1, 0, None), (3, 5, 6, None), (2, 8, 0, 9), (33, 4, 3, 8), (2, 3, 1, 30)])
def test_against_the_general_kernels(hd, batch, heads, pos, offset):
    g = torch.Generator(device="cuda").manual_seed(hd + heads)
    D, S = heads * hd, 12
    wide = torch.randn(batch, 3 * D + 8, device="cuda", generator=g).bfloat16()
    qkv, ref = wide.clone()[:, : 3 * D], wide.clone()[:, : 3 * D]
    kc = torch.randn(batch, heads, S, hd, device="cuda", generator=g).bfloat16()
    vc = torch.randn(batch, heads, S, hd, device="cuda", generator=g).bfloat16()
    k1, v1, k2, v2 = kc.clone(), vc.clone(), kc.clone(), vc.clone()
    dev = None if offset is None else torch.full((1,), offset, dtype=torch.int32, device="cuda")
    K.rope_kv_append(qkv, k1, v1, pos, 1e4, pos_dev=dev)
    K.rope_(ref[:, : 2 * D], 2 * heads, hd, 1, pos_offset=pos, theta=1e4, pos_dev=dev)
    K.kv_append(ref[:, D:2 * D], ref[:, 2 * D:], k2, v2, batch, 1, pos, pos_dev=dev)      # drops a token that does not fit (the last case)
    assert torch.equal(qkv, ref) and torch.equal(k1, k2) and torch.equal(v1, v2)
    if pos + (offset or 0) >= S:
        assert torch.equal(k1, kc) and torch.equal(v1, vc)


@pytest.mark.parametrize("hd", [64, 128])
def test_attention_of_one_piece(hd):
    # as many (row, head) pairs as need no split of the positions: the result leaves the kernel without a merge
    batch, heads, S, n = 40, 16, 200, 131
    g = torch.Generator(device="cuda").manual_seed(hd)
    q = torch.randn(batch, heads * hd, device="cuda", generator=g).bfloat16()
    kc = torch.randn(batch, heads, S, hd, device="cuda", generator=g).bfloat16()
    vc = torch.randn(batch, heads, S, hd, device="cuda", generator=g).bfloat16()
    out = K.decode_attn(q, kc, vc, n)
    kd, vd = kc[:, :, :n].double(), vc[:, :, :n].double()
    p = torch.softmax(q.double().view(batch, heads, 1, hd) @ kd.transpose(-1, -2) * hd ** -0.5, -1)
    want = (p @ vd).reshape(batch, heads * hd)
    assert K.decode_attn_splits(batch * heads, S) == 1
    assert float((out.double() - want).norm() / want.norm()) <= 2.0 ** -8      # one rounding to bf16
