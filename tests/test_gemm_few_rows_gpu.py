"""The product for a handful of rows against 64-bit sums: row counts at the padding edges, ragged widths, every cluster size."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 3, 16, 17, 32, 40, 48, 49, 64, 65])
@pytest.mark.parametrize("n,k", [(264, 512), (1024, 520), (4096, 4096), (11008, 1024), (32000, 576), (40008, 512)])
def test_few_rows(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m * 131 + n + k)
    x = torch.randn(m, k + 8, device="cuda", generator=g).bfloat16()[:, :k]      # a pitch that is not the width
    w = (torch.randn(n, k, device="cuda", generator=g) / k ** 0.5).bfloat16()
    bias = torch.randn(n, device="cuda", generator=g).bfloat16()
    res = torch.randn(m, n, device="cuda", generator=g).bfloat16()
    v = x.double() @ w.double().t()
    # an fp32 sum of k products and one rounding to bf16: its 2-norm is below the 2^-8 of the worst single value; 2^-9 on average
    cases = [(K.gemm(x, w), v, 2.0 ** -9), (K.gemm(x, w, out_dtype=torch.float32, alpha=0.5), 0.5 * v, 2e-6),
             (K.gemm(x, w, bias=bias, residual=res), v + bias.double() + res.double(), 2.0 ** -9),
             (K.gemm(x, w, bias=bias, act=K.ACT_RELU), torch.relu(v + bias.double()), 2.0 ** -9),
             (K.gemm(x, w, act=K.ACT_SILU), v * torch.sigmoid(v), 2.0 ** -8),
             (K.gemm(x, w, act=K.ACT_GELU), torch.nn.functional.gelu(v, approximate="tanh"), 2.0 ** -7)]   # tanh.approx: 2^-11 of 1
    for got, ref, tol in cases:
        assert float((got.double() - ref).norm() / ref.norm()) <= tol
    torch.cuda.synchronize()
    K.check_status()
