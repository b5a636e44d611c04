"""The 16-byte forms of the Mamba-3 convolution and gated norm against 64-bit statements."""
import pytest
import torch

from device_time import graph_us
from oa_b200 import _native as N
from oa_b200.ops import kernels as K
from oa_b200.ops import mamba3 as M3

pytestmark = pytest.mark.gpu


def _rel(a, e):
    return float((a.double().cpu() - e.double().cpu()).norm() / e.double().norm().cpu().clamp_min(1e-30))


# bf16: one rounding of each result (2^-8 at most); 1e-5 for the fp32 sums over rows
@pytest.mark.parametrize("kw", [2, 4])
@pytest.mark.parametrize("B,L,C,col0,tail", [(1, 1, 8, 0, 0), (2, 17, 40, 8, 16), (1, 130, 1032, 16, 8), (3, 64, 24, 3, 5),
                                               (2, 47, 40, 8, 0), (1, 48, 1032, 0, 8), (70, 17, 1040, 8, 8), (1000, 8, 1056, 0, 0), (520, 1, 768, 8, 0)])
def test_convolution(B, L, C, col0, tail, kw):
    g = torch.Generator(device="cuda").manual_seed(L + C)
    ld, rows = col0 + C + tail, B * L
    x = torch.randn(rows, ld, device="cuda", generator=g).bfloat16()
    w = torch.randn(kw, C, device="cuda", generator=g)
    lib, st = N.require(), N.stream()
    y, saved = x.clone(), torch.empty(rows, C, dtype=torch.bfloat16, device="cuda")
    assert lib.oa_mamba3_conv_fwd(1, y.data_ptr(), ld, col0, saved.data_ptr(), w.data_ptr(), B, L, C, kw, st) == 0
    xin = x[:, col0:col0 + C].double().reshape(B, L, C).requires_grad_(True)
    wd = w.double().requires_grad_(True)
    pad = torch.nn.functional.pad(xin, (0, 0, kw - 1, 0))
    ref = torch.nn.functional.silu(sum(pad[:, kw - 1 - j:kw - 1 - j + L] * wd[j] for j in range(kw)))
    assert torch.equal(saved, x[:, col0:col0 + C])
    assert torch.equal(y[:, :col0], x[:, :col0]) and torch.equal(y[:, col0 + C:], x[:, col0 + C:])
    assert _rel(y[:, col0:col0 + C], ref.reshape(rows, C)) <= 2.0 ** -8
    dy = torch.randn(rows, ld, device="cuda", generator=g).bfloat16()
    d, gbuf = dy.clone(), torch.empty(rows, C, dtype=torch.bfloat16, device="cuda")
    parts = torch.empty(B * ((L + 63) // 64), kw * C, device="cuda")
    assert lib.oa_mamba3_conv_bwd(1, d.data_ptr(), ld, col0, saved.data_ptr(), w.data_ptr(), parts.data_ptr(), gbuf.data_ptr(), B, L, C, kw, st) == 0
    dx, dw = torch.autograd.grad(ref, (xin, wd), dy[:, col0:col0 + C].double().reshape(B, L, C))
    assert _rel(d[:, col0:col0 + C], dx.reshape(rows, C)) <= 2.0 ** -7          # the gate's gradient is rounded too
    assert _rel(parts.sum(0).reshape(kw, C), dw) <= 2.0 ** -8
    assert torch.equal(d[:, :col0], dy[:, :col0]) and torch.equal(d[:, col0 + C:], dy[:, col0 + C:])


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2.0 ** -8), (torch.float32, 4e-6)])
@pytest.mark.parametrize("rows,H,P,extra", [(1, 1, 8, 8), (33, 3, 64, 0), (70, 48, 64, 24), (40, 5, 128, 8), (37, 7, 24, 8), (9, 3, 16, 3),
                                            (2801, 48, 64, 8), (8201, 8, 128, 0), (2750, 96, 32, 16), (5470, 24, 64, 3)])
def test_gated_norm(dtype, tol, rows, H, P, extra):
    g = torch.Generator(device="cuda").manual_seed(rows + P)
    d = M3.Mamba3Dims(H * P, H, P, 8, 0, has_z=False)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    y, proj, w, do = r(rows, H * P).to(dtype), r(rows, H * P + extra).to(dtype), 1 + 0.1 * r(H, P), r(rows, H * P).to(dtype)
    out, rstd = M3.gated_norm_fwd(y, proj, w, d)
    yd, zd, wd = y.double().requires_grad_(True), proj[:, :H * P].double().requires_grad_(True), w.double().requires_grad_(True)
    y3 = yd.reshape(rows, H, P)
    ref = (y3 * torch.rsqrt((y3 * y3).mean(-1, keepdim=True) + 1e-5) * wd).reshape(rows, H * P) * torch.nn.functional.silu(zd)
    assert _rel(out, ref) <= tol
    dproj = torch.full_like(proj, 3.0)
    dy, dw = M3.gated_norm_bwd(y, proj, w, rstd, do, d, dproj)
    gy, gz, gw = torch.autograd.grad(ref, (yd, zd, wd), do.double())
    assert _rel(dy, gy) <= tol and _rel(dproj[:, :H * P], gz) <= tol
    assert _rel(dw, gw.reshape(-1)) <= 1e-5
    assert bool((dproj[:, H * P:] == 3.0).all())


# A handful of tokens: the backward pass is a few microseconds like the forward pass, not a serial walk over 32 tokens.
def test_gated_norm_few_tokens():
    rows, H, P = 128, 8, 64
    d = M3.Mamba3Dims(H * P, H, P, 8, 0, has_z=False)
    y, proj, do, dproj = (torch.randn(rows, H * P, device="cuda").bfloat16() for _ in range(4))
    w = torch.ones(H, P, device="cuda")
    _, rstd = M3.gated_norm_fwd(y, proj, w, d)
    assert graph_us(*[lambda: M3.gated_norm_bwd(y, proj, w, rstd, do, d, dproj)] * 10) <= 5 * graph_us(*[lambda: M3.gated_norm_fwd(y, proj, w, d)] * 10)


# Sixteen tokens of the convolution take little more than their copy, whichever kernel runs them.
def test_convolution_few_tokens():
    L, C = 16, 768
    x, saved, w = torch.randn(L, C, device="cuda").bfloat16(), torch.empty(L, C, dtype=torch.bfloat16, device="cuda"), torch.randn(4, C, device="cuda")
    lib, y = N.require(), x.clone()

    def conv(rows):
        y.copy_(x)
        assert lib.oa_mamba3_conv_fwd(1, y.data_ptr(), C, 0, saved.data_ptr(), w.data_ptr(), 1, rows, C, 4, N.stream()) == 0

    one, all_ = graph_us(*[lambda: conv(1)] * 10), graph_us(*[lambda: conv(L)] * 10)
    assert all_ <= 2.8 * one                                 # 9.6 against 3.9 us; 15.6 with eight columns to a thread
