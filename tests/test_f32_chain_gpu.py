"""The short fp32 launches that may start under their predecessors, chained as a small model's step chains them: a replayed graph, in
which they overlap, gives what the same calls give one by one, also right after a kernel has changed what the first of them reads."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,seq,heads", [(1, 16, 1), (3, 40, 2), (16, 128, 4)])
def test_chain_in_a_graph(batch, seq, heads):
    hd, rows, vocab = 32, batch * seq, 96
    D = heads * hd
    g = torch.Generator(device="cuda").manual_seed(rows)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g) / s[-1] ** 0.5
    table, pos, qkv_w, up, down, head = r(vocab, D) * D ** 0.5, r(seq, D), r(3 * D, D), r(4 * D, D), r(D, 4 * D), r(vocab, D)
    ub, db = r(4 * D), r(D)
    gain, shift = 1 + 0.1 * r(D), 0.1 * r(D)
    ids = torch.randint(0, vocab, (rows,), device="cuda", generator=g, dtype=torch.int32)
    targets = torch.randint(0, vocab, (rows,), device="cuda", generator=g, dtype=torch.int32)
    attn = (batch, seq, heads, hd)

    def step():
        x = K.embedding_fwd(table, ids, pos, seq)
        h, mean, rstd = K.layernorm_fwd(x, gain, shift, 1e-5)
        qkv = K.gemm(h, qkv_w)
        parts = [qkv[:, i * D:(i + 1) * D] for i in range(3)]
        o, lse = K.flash_fwd(*parts, *attn)
        x1 = K.binary("add", x, o)
        z = torch.empty(rows, 4 * D, device="cuda")
        u = K.gemm(x1, up, bias=ub, act=K.ACT_GELU, aux_out=z)
        y = K.gemm(u, down, bias=db, residual=x1)
        logits = K.gemm(y, head)
        row_loss, dlogits = K.xent_fwd_bwd(logits, targets, grad_scale=1.0 / rows)
        loss = K.mean_f32(row_loss)
        dy = K.gemm(dlogits, head, b_mn=True)
        ddown, ddb = torch.empty_like(down), torch.empty_like(db)
        K.weight_grad(dy, u, out=ddown, accumulate=False, bias_out=ddb, bias_accumulate=False)
        dz = K.gemm(dy, down, b_mn=True, act=K.ACT_GELU_BWD, aux_in=z)
        dx1 = K.binary("add", dy, K.gemm(dz, up, b_mn=True))
        dq = K.flash_bwd(*parts, o, dx1, lse, *attn)
        dh = K.gemm(torch.cat(dq, 1), qkv_w, b_mn=True)
        dx, dgain, dshift = K.layernorm_bwd(x, gain, dh, mean, rstd)
        return [loss, dlogits, y, ddown, ddb, K.col_sum(dz), *dq, dx, dgain, dshift]

    step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    for _ in range(4):
        graph.replay()
        got = [t.clone() for t in out]
        torch.cuda.synchronize()
        want = step()
        for i, (a, b) in enumerate(zip(got, want)):
            assert torch.equal(a, b), i
        table.mul_(-0.75)
        qkv_w.add_(qkv_w, alpha=0.25)
    assert all(bool(torch.isfinite(t).all()) for t in got)
    K.check_status()
