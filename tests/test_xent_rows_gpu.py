"""Cross-entropy with the row on the chip: row lengths at the edges of the warp, shared-memory and general paths."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


# bf16: one rounding, at most 2^-8 of a value.  fp32: exp(x) as a power of two of x log2(e) carries the rounding of that product,
# 2^-24 |x| for |x| <= 30, the rounding of the log-sum-exp, and the 2^-22 of the power itself: 4e-6
@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2.0 ** -8), (torch.float32, 4e-6)])
@pytest.mark.parametrize("rows,vocab,ld", [(9, 8, 8), (13, 256, 256), (8, 1024, 1024), (5, 1032, 1032), (3, 8200, 8200), (4, 32000, 32000), (3, 32003, 32008),
                                           (2, 50257, 50264), (2, 51200, 51200), (2, 102400, 102400), (2, 102408, 102408), (6, 1000, 1001)])
@pytest.mark.parametrize("in_place", [False, True])
def test_cross_entropy_rows(dtype, tol, rows, vocab, ld, in_place):
    g = torch.Generator().manual_seed(vocab + rows)
    full = (3.0 * torch.randn(rows, ld, generator=g)).to(dtype)
    t = torch.randint(0, vocab, (rows,), generator=g, dtype=torch.int32)
    t[0], t[-1] = vocab - 1, -100
    if rows > 4:
        t[1] = vocab + 3                                     # out of range: NaN loss, softmax as gradient
        full[2, : vocab // 2] = float("-inf")                # masked half
        t[2] = vocab - 1
    dev = full.cuda()
    logits = dev[:, :vocab]
    out = logits if in_place else None
    if out is None:
        out = torch.full((rows, ld), 7.0, dtype=dtype, device="cuda")[:, :vocab]
    loss, d = K.xent_fwd_bwd(logits, t.cuda(), grad_scale=0.25, dlogits=out)
    lf = full[:, :vocab].double()
    lse = torch.logsumexp(lf, -1)
    p = torch.softmax(lf, -1)
    for r in range(rows):
        tr = int(t[r])
        if tr == -100:
            assert float(loss[r]) == 0.0 and not d[r].any()
            continue
        ref = p[r] * 0.25
        if tr < vocab:
            assert abs(float(loss[r]) - float(lse[r] - lf[r, tr])) <= 4e-6 * max(1.0, float(lse[r]))
            ref = ref.clone()
            ref[tr] -= 0.25
        else:
            assert torch.isnan(loss[r])
        # p - 1 cancels at a sure target, so the error is that of p itself
        assert float((d[r].double().cpu() - ref).norm() / torch.maximum(ref.norm(), 0.25 * p[r].norm())) <= tol
    if not in_place and ld > vocab:
        pad = out.as_strided((rows, ld - vocab), (ld, 1), out.storage_offset() + vocab)
        assert bool((pad == 7.0).all())
    loss2, none = K.xent_fwd_bwd(full.cuda()[:, :vocab], t.cuda())
    assert none is None
    torch.testing.assert_close(loss2, loss, rtol=0, atol=0, equal_nan=True)
