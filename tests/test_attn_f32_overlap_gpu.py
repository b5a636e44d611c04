"""fp32 attention gradients beside their neighbours in a stream: what comes before is read, what follows finds both done, eagerly and in a graph."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


# blocks for a part of the chip, on both sides of a full mask's lines and for several waves (both gradients in one launch, and in two), the last tile
# ragged, every split of a row, more sequences than a grid holds twice
@pytest.mark.parametrize("batch,seq,heads,hd", [(1, 33, 1, 32), (16, 128, 4, 32), (18, 128, 4, 32), (19, 128, 4, 32), (40, 128, 4, 64), (2, 515, 4, 64), (3, 200, 2, 128), (64, 160, 4, 20), (34, 130, 4, 64),
                                               (33000, 2, 1, 4)])
@pytest.mark.parametrize("causal", [False, True])
def test_neighbours_in_the_stream(batch, seq, heads, hd, causal):
    D, rows = heads * hd, batch * seq
    g = torch.Generator(device="cuda").manual_seed(seq + hd)
    r = lambda n: torch.randn(rows, n, device="cuda", generator=g)
    qkv, half = r(3 * D), 0.5 * r(D)
    parts = [qkv[:, i * D:(i + 1) * D] for i in range(3)]
    o, lse = K.flash_fwd(*parts, batch, seq, heads, hd, causal=causal)
    do = torch.empty_like(half)

    def step():
        do.copy_(K.binary("add", half, half))                      # the gradient is made by the launches just before
        dq, dk, dv = K.flash_bwd(*parts, o, do, lse, batch, seq, heads, hd, causal=causal)[:3]
        return [K.binary("add", t.contiguous(), half) for t in (dk, dv, dq)]

    step()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        kept = step()
    do.zero_()
    graph.replay()
    x = [p.reshape(batch, seq, heads, hd).transpose(1, 2).double().detach().requires_grad_() for p in parts]
    s = x[0] @ x[1].transpose(-1, -2) / hd ** 0.5
    if causal:
        s = s.masked_fill(torch.ones(seq, seq, device="cuda").triu(1).bool(), float("-inf"))
    (s.softmax(-1) @ x[2]).backward((half + half).double().reshape(batch, seq, heads, hd).transpose(1, 2))
    flat = lambda t: t.transpose(1, 2).reshape(rows, D) + half.double()
    want = [flat(x[i].grad) for i in (1, 2, 0)]
    for got in (kept, step()):
        for a, e in zip(got, want):
            # dot products and sums of at most 515 terms in 32 bits and __expf's few units in the last place of a probability
            assert float((a.double() - e).norm() / e.norm()) <= 1e-5
