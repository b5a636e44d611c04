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
    got = K.few_rows_step(x, w, residual=res, norm_w=nw)
    if got is None:                                         # left to the tile kernels
        assert K.few_rows_step(x, w) is None
        return
    out, out_w, sq = got
    y = x.double() @ w.double().t() + res.double()
    assert _rel(out, y) <= TOL
    assert torch.equal(out_w, (out.float() * nw.float()).bfloat16())
    assert _rel(sq.sum(0), (out.double() ** 2).sum(1)) <= 1e-5
    # the product behind: as if it had been given the normed rows
    w2, bias = (r(512, n) / n ** 0.5).bfloat16(), r(512).bfloat16()
    if K.few_rows_step(out_w[:, :n], w2) is not None:
        got2 = K.few_rows_step(out_w, w2, squares=sq, eps=1e-5, bias=bias)
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
    if got is None:
        assert K.few_rows_step(x, w) is None
        return
    z = x.double() @ w.double().t() * torch.rsqrt(sq.double().sum(0) / k + 1e-6)[:, None]
    assert got.shape == (m, f) and _rel(got, torch.nn.functional.silu(z[:, :f]) * z[:, f:]) <= TOL
    torch.cuda.synchronize()
    K.check_status()
