"""Attention at head dims 64 and 128: the exponentials that are worked out on the multiply-add pipe, masked and invalid scores, and rows that
end inside a group of four."""
import math

import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


def _split(qkv, hd, heads):
    D = heads * hd
    return qkv[:, :D], qkv[:, D:2 * D], qkv[:, 2 * D:]


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("seq", [127, 128, 129, 385, 1026])
def test_masked_values_do_not_leak(hd, seq):
    """Keys that the causal mask hides hold values of 1e38: a probability of anything but 0 would show."""
    heads, cut = 3, seq // 2
    g = torch.Generator(device="cuda").manual_seed(seq)
    qkv = torch.randn(seq, 3 * heads * hd, device="cuda", generator=g).bfloat16()
    big = qkv.clone()
    big[cut:, 2 * heads * hd:] = 1e38
    a, _ = K.flash_fwd(*_split(qkv, hd, heads), 1, seq, heads, hd, causal=True)
    b, _ = K.flash_fwd(*_split(big, hd, heads), 1, seq, heads, hd, causal=True)
    assert torch.equal(a[:cut], b[:cut])


@pytest.mark.parametrize("hd", [64, 128])
def test_exponentials_over_their_range(hd):
    """One key of value 1 among keys of value 0, at every distance below the row's maximum: the output is its probability, which 2^-n
    down to the smallest normal number takes through every exponent.  Each key position in turn, so that both pipes are met."""
    seq = 128
    gap = torch.linspace(0.0, 80.0, seq, device="cuda")                      # natural log units below the maximum, by query
    q = torch.zeros(seq, hd, device="cuda")
    q[:, 0], q[:, 1] = 1.0, gap
    for pos in range(1, 16):
        k, v = torch.zeros(seq, hd, device="cuda"), torch.zeros(seq, hd, device="cuda")
        k[pos, 1], v[pos, :] = -1.0, 1.0
        qb, kb, vb = q.bfloat16(), k.bfloat16(), v.bfloat16()
        o, lse = K.flash_fwd(qb, kb, vb, 1, seq, 1, hd, scale=1.0, causal=False)
        s = qb.double() @ kb.double().t()
        ref = torch.softmax(s, -1) @ vb.double()
        # a rounding to bf16 (eight significant bits) moves a single value by up to 2^-8 of itself; the probability and the output are
        # rounded once each, and a score of up to 80 has an error of 80 x 2^-23 in fp32
        assert float(((o.double() - ref).abs() / ref).max()) <= 2.0 ** -7 + 80 * 2.0 ** -23
        assert (lse.double()[0, 0] - torch.logsumexp(s, -1)).abs().max().item() <= 1e-6 * math.log(seq) + 1e-6


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
def test_invalid_scores_show(hd, bad):
    """A NaN or an infinity in one key reaches every row that looks at it, whichever pipe its exponential takes."""
    seq = 256
    g = torch.Generator(device="cuda").manual_seed(7)
    qkv = torch.rand(seq, 3 * hd, device="cuda", generator=g).bfloat16() + 0.5     # positive: an infinite key gives infinite scores
    for pos in (3, 10, 11, 66, 67, 130):
        x = qkv.clone()
        x[pos, hd] = bad
        o, _ = K.flash_fwd(*_split(x, hd, 1), 1, seq, 1, hd, causal=False)
        q, k, v = (t.double() for t in _split(x, hd, 1))
        ref = torch.softmax(q @ k.t() / hd ** 0.5, -1) @ v
        assert torch.equal(torch.isnan(o), torch.isnan(ref)), (pos, bad)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("batch,seq", [(2, 1), (2, 30), (2, 33), (3, 127), (2, 131), (2, 258), (1, 515)])
def test_backward_writes_its_rows_only(hd, causal, batch, seq):
    """Rows of one sequence end beside the next one's: gradients against 64 bits, and nothing beyond the last row."""
    heads = 2
    D = heads * hd
    g = torch.Generator(device="cuda").manual_seed(seq)
    qkv = torch.randn(batch * seq, 3 * D, device="cuda", generator=g).bfloat16()
    do = torch.randn(batch * seq, D, device="cuda", generator=g).bfloat16()
    o, lse = K.flash_fwd(*_split(qkv, hd, heads), batch, seq, heads, hd, causal=causal)
    room = torch.full((batch * seq + 8, 3 * D), 7.0, device="cuda", dtype=torch.bfloat16)
    K.flash_bwd(*_split(qkv, hd, heads), o, do, lse, batch, seq, heads, hd, causal=causal, dqkv=room[:batch * seq])
    x = qkv.double().requires_grad_(True)
    q, k, v = (t.reshape(batch, seq, heads, hd).transpose(1, 2) for t in _split(x, hd, heads))
    s = q @ k.transpose(-1, -2) / hd ** 0.5
    if causal:
        s = s.masked_fill(~torch.ones(seq, seq, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    ref, = torch.autograd.grad((torch.softmax(s, -1) @ v).transpose(1, 2).reshape(batch * seq, D), x, do.double())
    # probabilities, their gradients, the output of the forward pass and the results are rounded to bf16: in the norm up to 2^-9 each
    for i in range(3):
        e, r = room[:batch * seq, i * D:(i + 1) * D].double() - ref[:, i * D:(i + 1) * D], ref[:, i * D:(i + 1) * D]
        assert float(e.norm()) <= 2.0 ** -7 * float(r.norm()) + 1e-2 * (seq == 1)
    assert bool((room[batch * seq:] == 7.0).all())
    torch.cuda.synchronize()
    K.check_status()
