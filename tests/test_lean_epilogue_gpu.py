"""Products that are only scaled, rounded to bf16 and stored through TMA: batched ones with a factor, and the grouped ones of the
mixture of experts, at both tile widths, with ragged rows and columns, every operand layout and a group without rows."""
import pytest
import torch

from oa_b200.ops import kernels as K
from oa_b200.ops import moe as M

pytestmark = pytest.mark.gpu

# one rounding to bf16 (2^-9 of a value at most) of fp32 sums of exact products
TOL = 2.0 ** -8


def _rel(got, ref):
    return float((got.double() - ref).norm() / ref.norm())


@pytest.fixture(autouse=True)
def _status():
    yield
    torch.cuda.synchronize()
    K.check_status()


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("nb,m,n,k", [(2, 40, 72, 96), (5, 200, 136, 72), (64, 200, 520, 64), (150, 128, 256, 8)])
@pytest.mark.parametrize("alpha", [1.0, -0.375])
def test_batched(nb, m, n, k, a_mn, b_mn, alpha):
    g = torch.Generator(device="cuda").manual_seed(m + n)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    a, b = r(nb, k, m) if a_mn else r(nb, m, k), r(nb, k, n) if b_mn else r(nb, n, k)
    buf = torch.full((nb, m + 3, n + 8), 7.0, device="cuda").bfloat16()
    out = buf[:, :m, :n]
    K.bgemm(a, b, a_mn=a_mn, b_mn=b_mn, out=out, alpha=alpha)
    ref = alpha * ((a.transpose(1, 2) if a_mn else a).double() @ (b if b_mn else b.transpose(1, 2)).double())
    assert _rel(out, ref) <= TOL
    out.fill_(7.0)
    assert bool((buf == 7.0).all())                             # nothing beyond the last row and column


@pytest.mark.parametrize("n,k", [(72, 136), (136, 520), (520, 264), (256, 128)])
def test_grouped(n, k):
    g = torch.Generator(device="cuda").manual_seed(n + k)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    tokens, experts = 500, 5
    idx = torch.randint(0, experts - 1, (tokens, 2), device="cuda", generator=g, dtype=torch.int32)
    idx[idx == 2] = experts - 1                                 # expert 2 has no rows
    plan = M.plan(idx, experts)
    offs = plan.offsets.tolist()
    assert offs[2] == offs[3] and offs[-1] < plan.max_rows
    x, dy = M.gather(r(tokens, k), plan), M.gather(r(tokens, n), plan)
    w = r(experts, n, k)
    nan = lambda *s: torch.full(s, float("nan"), device="cuda").bfloat16()
    y = M.grouped_linear(x, w, None, plan, out=nan(plan.max_rows, n))
    dx = M.grouped_linear(dy, w, None, plan, b_mn=True, out=nan(plan.max_rows, k))
    dw = M.grouped_weight_grad(dy, x, plan, out=nan(experts, n, k))
    for e in range(experts):
        s = slice(offs[e], offs[e + 1])
        if e == 2:
            assert not bool(dw[e].any())                        # zeros, not what was there
            continue
        assert _rel(y[s], x[s].double() @ w[e].double().t()) <= TOL
        assert _rel(dx[s], dy[s].double() @ w[e].double()) <= TOL
        assert _rel(dw[e], dy[s].double().t() @ x[s].double()) <= TOL
    assert bool(y[offs[-1]:].isnan().all()) and bool(dx[offs[-1]:].isnan().all())
