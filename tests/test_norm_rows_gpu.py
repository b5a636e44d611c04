"""RMSNorm kernels with the row on the chip: row widths around the 256-column pieces of a warp and the splits over warps."""
import pytest
import torch

from device_time import graph_us
from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


def _rel(got, ref):
    ref = ref.double()
    return float((got.double().cpu() - ref).norm() / ref.norm().clamp_min(1e-30))


# bf16 keeps 8 significant bits: one rounding changes a value by at most 2^-8 of it, and so the 2-norm
@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2.0 ** -8), (torch.float32, 2e-6)])
@pytest.mark.parametrize("rows,cols", [(1, 8), (7, 248), (33, 256), (5, 264), (300, 1024), (9, 1032), (1201, 1536), (17, 2048), (3, 2056), (130, 4096), (6, 4104),
                                       (1185, 2056), (1185, 2880), (2369, 1032), (40, 512), (25, 768), (1300, 1024), (1184, 1024)])
def test_rmsnorm_forward_and_backward(dtype, tol, rows, cols):
    g = torch.Generator().manual_seed(rows * 10007 + cols)
    x, dy, res, dres = (torch.randn(rows, cols, generator=g).to(dtype) for _ in range(4))
    w = (1.0 + 0.1 * torch.randn(cols, generator=g)).to(dtype)
    c = lambda t: t.cuda()
    for r in (None, res):
        y, rstd, s = K.rmsnorm_fwd(c(x), c(w), 1e-5, residual=None if r is None else c(r))
        yr, rr, sr = K.rmsnorm_fwd(x.float(), w.float(), 1e-5, residual=None if r is None else r.float())
        if r is not None:
            assert _rel(s, sr) <= tol
        assert _rel(rstd, rr) <= 2e-6
        assert _rel(y, yr) <= 3 * tol                       # a residual's sum is rounded first, here and in the reference: up to three roundings
    _, rstd, _ = K.rmsnorm_fwd(c(x), c(w), 1e-5)
    xd, wd, dd = x.double(), w.double(), dy.double()
    xh = xd * rstd.double().cpu()[:, None]
    gw = dd * wd
    dx0 = rstd.double().cpu()[:, None] * (gw - xh * (gw * xh).mean(-1, keepdim=True))
    for r in (None, dres):
        dx, dw = K.rmsnorm_bwd(c(x), c(w), c(dy), rstd, dres=None if r is None else c(r))
        assert _rel(dx, dx0 if r is None else dx0 + r.double()) <= tol
        assert _rel(dw, (dd * xh).sum(0)) <= tol
        acc = torch.ones(cols, dtype=torch.float32, device="cuda")
        K.rmsnorm_bwd(c(x), c(w), c(dy), rstd, dw_out=acc, accumulate_dw=True)
        assert _rel(acc, (dd * xh).sum(0) + 1.0) <= 1e-5    # fp32 sums of up to 2369 rows
    torch.cuda.synchronize()


# A row that just fits the registers takes no longer than one that just does not: 4736 x 4096 with a residual took 1.6 times as long.
@pytest.mark.parametrize("rows,cols,dtype", [(4736, 4096, torch.bfloat16), (4736, 2880, torch.bfloat16), (9472, 2048, torch.float32)])
def test_wide_rows_with_a_residual(rows, cols, dtype):
    def us(c):
        x, w, r = (torch.randn(*s, device="cuda").to(dtype) for s in ((rows, c), (c,), (rows, c)))
        return graph_us(*[lambda: K.rmsnorm_fwd(x, w, 1e-5, residual=r)] * 10) / (rows * c)

    assert us(cols) <= 1.3 * us(4104 if dtype == torch.bfloat16 else 2056)
