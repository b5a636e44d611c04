"""The product for a handful of rows against 64-bit sums: row counts at the padding edges, ragged widths, cluster sizes 1, 2, 4 and 8 with
even and uneven shares of K, several waves of tiles."""
import pytest
import torch

from device_time import graph_us
from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 3, 16, 17, 32, 40, 48, 49, 64, 65])
@pytest.mark.parametrize("n,k", [(264, 512), (1024, 520), (4096, 4096), (11008, 1024), (32000, 576), (40008, 512),
                                   (8192, 1096), (2048, 2120), (11008, 1048), (40008, 1032)])
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

# The line between this kernel and the tile kernel lies where neither is much slower; weights come from memory (8 x 51 MB).
@pytest.mark.parametrize("m,n,k", [(64, 50264, 512), (64, 38016, 1024), (48, 128256, 512), (16, 50264, 512), (1, 50264, 512), (64, 14336, 512),
                                   (48, 12288, 768)])
def test_not_slower_than_the_tile_kernel(m, n, k):
    ws = [torch.randn(n, k, device="cuda").bfloat16() for _ in range(max(1, -(-400_000_000 // (n * k * 2))))]
    x, out = torch.randn(m, k, device="cuda").bfloat16(), torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
    tiled = min(graph_us(*[lambda w=w, bn=bn: K.gemm(x, w, out=out, force_bn=bn) for w in ws]) for bn in (128, 256))
    assert graph_us(*[lambda w=w: K.gemm(x, w, out=out) for w in ws]) <= 1.15 * tiled
