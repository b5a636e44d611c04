"""bf16 products with fp32 results, and those summed from fp32 partial products: stores that cover eight rows at a time, at rows and columns off
the tiles, added to what is there, into a wider matrix."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(8, 8, 64), (264, 520, 128), (3000, 1000, 520), (2888, 2056, 72), (1024, 1024, 8192), (520, 264, 16384)])
@pytest.mark.parametrize("kind", ["fp32", "add", "split"])
def test_rows(m, n, k, kind):
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a, b = (torch.randn(k, s, device="cuda", generator=g).bfloat16() for s in (m, n))
    ref = a.double().t() @ b.double()
    if kind == "split":                                    # a long reduction is cut into fp32 partial products
        assert float((K.gemm(a, b, a_mn=True, b_mn=True).double() - ref).norm() / ref.norm()) <= 2.0 ** -8
    else:
        room = torch.randn(m + 5, n + 8, device="cuda", generator=g)
        before = room.clone()
        K.gemm(a, b, a_mn=True, b_mn=True, out=room[:m, :n], accumulate=kind == "add")
        want = ref + (before[:m, :n].double() if kind == "add" else 0)
        # sums of k exact products in fp32: errors of 2^-24 of partial sums, which grow like the square root of their number
        assert float((room[:m, :n].double() - want).norm() / want.norm()) <= 2.0 ** -24 * 4 * k ** 0.5
        room[:m, :n] = before[:m, :n]
        assert torch.equal(room, before)                   # nothing beyond the last row and column
    torch.cuda.synchronize()
    K.check_status()
