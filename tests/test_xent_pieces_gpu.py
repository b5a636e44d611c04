"""Cross-entropy with the row in shared memory, with a running maximum per thread."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
LOWEST = float(torch.finfo(torch.bfloat16).min)


# one vector per thread and several, an odd number of vectors, a remainder off the vectors
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("vocab", [4104, 4112, 8192, 16392, 20003, 32008])
@pytest.mark.parametrize("kind", ["random", "rising", "falling", "masked"])
def test_row(vocab, kind, dtype):
    rows = 5
    ld = (vocab + 7) // 8 * 8
    g = torch.Generator(device="cuda").manual_seed(vocab)
    x = torch.randn(rows, ld, device="cuda", generator=g) * 3
    if kind in ("rising", "falling"):                      # the maximum moves with every vector, or never
        x += torch.linspace(-60, 60, ld, device="cuda") * (1 if kind == "rising" else -1)
    t = torch.randint(0, vocab // 2, (rows,), device="cuda", dtype=torch.int32, generator=g)
    if kind == "masked":                                   # half of the row is hidden, by an infinity and by the type's lowest value
        x[:, vocab // 2:3 * vocab // 4] = float("-inf")
        x[:, 3 * vocab // 4:] = LOWEST
        x[4, :] = LOWEST                                   # all of it: every entry is as likely
    x = x.to(dtype)
    d = torch.zeros_like(x)
    loss, d = K.xent_fwd_bwd(x[:, :vocab], t, grad_scale=0.5, dlogits=d[:, :vocab])
    r = x[:, :vocab].double()
    lse = torch.logsumexp(r, 1)
    ref = lse - r.gather(1, t.long()[:, None])[:, 0]
    grad = (torch.exp(r - lse[:, None]) - torch.nn.functional.one_hot(t.long(), vocab)) * 0.5
    if kind == "masked":                                   # in fp32 log(vocab) is lost beside the lowest value: every entry counts as 1
        other = torch.ones(vocab, dtype=torch.bool, device="cuda")
        other[t[4].long()] = False
        assert float(loss[4]) == 0.0 and bool((d[4][other] == 0.5).all()) and float(d[4, t[4].long()]) == 0.0
        ref, grad, loss, d = ref[:4], grad[:4], loss[:4], d[:4]
    # exponentials to 2^-22 and sums of as many terms in fp32; the gradient is rounded to its type
    assert float(((loss.double() - ref).abs() / ref.abs().clamp_min(1.0)).max()) <= 2e-6
    assert float((d.double() - grad).norm() / grad.norm()) <= (2.0 ** -9 if dtype == torch.bfloat16 else 2e-6)
    if kind == "masked":
        assert bool((d[:, vocab // 2:] == 0).all())
