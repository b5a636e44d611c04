"""LayerNorm backward that adds the residual stream's gradient, and one launch for both parameter sums, against 64 bits."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


# one row, fewer rows than a block has warps, rows off the grid; the narrowest row, one off the warp's step, several steps; few and many partial rows
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", [(1, 8), (5, 264), (1027, 256), (4096, 1032)])
@pytest.mark.parametrize("with_dres", [False, True])
def test_against_64_bits(rows, cols, dtype, with_dres):
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dtype)
    x, w, dy, dres = r(rows, cols), 1 + 0.1 * r(cols), r(rows, cols), 3 * r(rows, cols)
    _, mean, rstd = K.layernorm_fwd(x, w, None, 1e-5)
    seed = torch.randn(2, cols, device="cuda", generator=g)
    dw, db = seed[0].clone(), seed[1].clone()
    dx, dw, db = K.layernorm_bwd(x, w, dy, mean, rstd, dres=dres if with_dres else None, dw_out=dw, db_out=db, accumulate=True)
    xd, wd, dd = x.double(), w.double(), dy.double()
    xh = (xd - mean.double()[:, None]) * rstd.double()[:, None]
    t = dd * wd
    want = rstd.double()[:, None] * (t - t.mean(1, keepdim=True) - xh * (t * xh).mean(1, keepdim=True))
    if with_dres:
        want = want + dres.double()
    # one rounding of the result (2^-8 of an element is bf16's spacing), or a few dozen fp32 operations in a row's sums
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 64 * 2.0 ** -24
    assert float((dx.double() - want).abs().max()) <= tol * float(want.abs().max())
    # the sums over rows stay in 32 bits: a sequence of at most `rows` additions per thread and of the threads' parts
    for got, ref in ((dw, seed[0].double() + (dd * xh).sum(0)), (db, seed[1].double() + dd.sum(0))):
        assert float((got.double() - ref).abs().max()) <= 64 * 2.0 ** -24 * (1 + float(dd.abs().sum(0).max()))
