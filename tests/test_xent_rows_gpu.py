"""Cross-entropy with the row on the chip: row lengths at the edges of the warp, shared-memory and general paths."""
import pytest
import torch

from device_time import graph_us
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


# More rows than SMs, where the loss alone and the gradient may take different kernels; masks of -inf and of the type's lowest value.
@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2.0 ** -8), (torch.float32, 4e-6)])
@pytest.mark.parametrize("rows,vocab,ld", [(150, 16384, 16384), (151, 16392, 16392), (149, 57344, 57344), (149, 57352, 57352), (160, 999, 1001)])
def test_many_rows(dtype, tol, rows, vocab, ld):
    g = torch.Generator().manual_seed(vocab)
    full = (3.0 * torch.randn(rows, ld, generator=g)).to(dtype)
    low = torch.finfo(dtype).min
    full[0, : vocab // 2] = float("-inf")
    full[1, : vocab // 2] = low
    full[2, : vocab - 1] = low
    t = torch.randint(vocab // 2, vocab, (rows,), generator=g, dtype=torch.int32)
    t[2] = vocab - 1
    out = torch.empty(rows, ld, dtype=dtype, device="cuda")[:, :vocab]
    loss, d = K.xent_fwd_bwd(full.cuda()[:, :vocab], t.cuda(), grad_scale=0.25, dlogits=out)
    alone, _ = K.xent_fwd_bwd(full.cuda()[:, :vocab], t.cuda())
    lf = full[:, :vocab].double()
    lse = torch.logsumexp(lf, -1)
    ref = lse - lf.gather(1, t.long()[:, None])[:, 0]
    for got in (loss, alone):
        assert bool(((got.double().cpu() - ref).abs() <= 4e-6 * lse.abs().clamp_min(1.0)).all())
    p = torch.softmax(lf, -1) * 0.25
    grad = p.clone()
    grad.scatter_add_(1, t.long()[:, None], torch.full((rows, 1), -0.25, dtype=torch.float64))
    err = (d.double().cpu() - grad).norm(dim=1) / torch.maximum(grad.norm(dim=1), p.norm(dim=1))
    assert float(err.max()) <= tol


def test_the_loss_alone_reads_as_fast_as_it_may():
    x = torch.randn(4096, 32000, device="cuda")
    t = torch.randint(0, 32000, (4096,), device="cuda", dtype=torch.int32)
    d = torch.empty_like(x)
    # it moves half the bytes of loss and gradient; with the row in shared memory it took 0.6 of their time
    assert graph_us(*[lambda: K.xent_fwd_bwd(x, t)] * 4) <= 0.52 * graph_us(*[lambda: K.xent_fwd_bwd(x, t, grad_scale=1.0, dlogits=d)] * 4)


# Logits that are columns of a wider matrix: the gradient made for them has their pitch, one of another pitch is refused.
def test_pitch():
    full = torch.randn(6, 40, device="cuda")
    t = torch.arange(6, device="cuda", dtype=torch.int32)
    x = full[:, :33]
    loss, d = K.xent_fwd_bwd(x, t, grad_scale=1.0)
    ref = torch.softmax(x.double(), -1) - torch.nn.functional.one_hot(t.long(), 33)
    assert d.shape == x.shape and float((d.double() - ref).norm() / ref.norm()) <= 4e-6
    with pytest.raises(ValueError):
        K.xent_fwd_bwd(x, t, grad_scale=1.0, dlogits=torch.empty(6, 33, device="cuda"))
    loss1, d1 = K.xent_fwd_bwd(x[:1], t[:1], grad_scale=1.0, dlogits=torch.empty(1, 33, device="cuda"))
    assert torch.equal(d1[0], d[0]) and torch.equal(loss1[0], loss[0])
