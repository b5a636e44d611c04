"""Few-row products that carry the RMS norms around them, and the gated one, against 64 bits."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu

# an operand, or a row times the norm's weight, rounded to bf16 once and the result once: in the norm 2^-9 each
TOL = 2.0 ** -8


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm())


# clusters of one to eight, columns and reductions off the tiles, every number of row groups
@pytest.mark.parametrize("m", [1, 3, 16, 17, 40, 64])
@pytest.mark.parametrize("n,k", [(256, 512), (264, 520), (4096, 1024), (9480, 4104), (20000, 4096)])
def test_norm_behind_and_in_front(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m + n)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w, res, nw = r(m, k).bfloat16(), (r(n, k) / k ** 0.5).bfloat16(), (3 * r(m, n)).bfloat16(), (1 + 0.2 * r(n)).bfloat16()
    out, out_w, sq = K.few_rows_step(x, w, residual=res, norm_w=nw)      # all of these are the few-row kernel's
    y = x.double() @ w.double().t() + res.double()
    assert _rel(out, y) <= TOL
    assert torch.equal(out_w, (out.float() * nw.float()).bfloat16())
    assert _rel(sq.sum(0), (out.double() ** 2).sum(1)) <= 1e-5
    # the product behind: as if it had been given the normed rows
    w2, bias = (r(512, n) / n ** 0.5).bfloat16(), r(512).bfloat16()
    got2 = K.few_rows_step(out_w, w2, squares=sq, eps=1e-5, bias=bias)
    assert (got2 is None) == (n < 512)                       # reductions too short for it
    if got2 is not None:
        o = out.double()
        normed = o * torch.rsqrt((o * o).mean(1, keepdim=True) + 1e-5) * nw.double()
        assert _rel(got2, normed @ w2.double().t() + bias.double()) <= TOL
    torch.cuda.synchronize()
    K.check_status()


@pytest.mark.parametrize("m", [1, 16, 33, 64])
@pytest.mark.parametrize("f,k", [(128, 512), (200, 520), (1408, 2048), (11008, 4096), (4104, 1024)])
def test_gated(m, f, k):
    g = torch.Generator(device="cuda").manual_seed(m + f)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w, sq = r(m, k).bfloat16(), (r(2 * f, k) / k ** 0.5).bfloat16(), r(3, m).abs()
    got = K.few_rows_step(x, w, squares=sq, eps=1e-6, gated=True)
    z = x.double() @ w.double().t() * torch.rsqrt(sq.double().sum(0) / k + 1e-6)[:, None]
    assert got.shape == (m, f) and _rel(got, torch.nn.functional.silu(z[:, :f]) * z[:, f:]) <= TOL
    torch.cuda.synchronize()
    K.check_status()


# short reductions, few columns, many rows, wide and shallow weights for many rows (on 148 SMs), weights in another order
@pytest.mark.parametrize("m,n,k", [(1, 512, 504), (1, 248, 512), (65, 512, 512), (64, 12288, 512), (33, 40960, 2048)])
def test_left_to_others(m, n, k):
    x, w = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(n, k, device="cuda").bfloat16()
    assert K.few_rows_step(x, w) is None
    assert K.few_rows_step(x, torch.randn(k, 1024, device="cuda").bfloat16().t()) is None
