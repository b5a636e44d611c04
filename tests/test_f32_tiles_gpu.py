"""fp32 products through the tile kernel and its epilogue."""
import pytest
import torch

from device_time import graph_us
from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


def _gelu(z):
    return torch.nn.functional.gelu(z, approximate="tanh")


# fp32 sums of up to 2048 products of unit variance in any order: a few 2^-24 sqrt(K), below 2e-6 of the result's norm
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (4, 4, 4), (65, 36, 20), (64, 64, 16), (132, 68, 100), (2048, 384, 128), (128, 512, 2048), (96, 200, 516), (33, 65, 17)])
def test_products(m, n, k, a_mn, b_mn):
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n * 3 + k)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    a, b = r(k, m) if a_mn else r(m, k), r(k, n) if b_mn else r(n, k)
    v = (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double()
    bias, res, z, old = r(n), r(m, n), r(m, n), r(m, n)
    rel = lambda got, ref: float((got.double() - ref).norm() / ref.norm().clamp_min(1e-30))
    kw = dict(a_mn=a_mn, b_mn=b_mn)
    assert rel(K.gemm(a, b, **kw), v) <= 2e-6
    assert rel(K.gemm(a, b, alpha=0.5, out=old.clone(), accumulate=True, **kw), 0.5 * v + old.double()) <= 2e-6
    assert rel(K.gemm(a, b, bias=bias, residual=res, **kw), v + bias.double() + res.double()) <= 2e-6
    aux = torch.empty(m, n, device="cuda")
    h = K.gemm(a, b, bias=bias, act=K.ACT_GELU, aux_out=aux, **kw)
    assert rel(aux, v + bias.double()) <= 2e-6 and rel(h, _gelu(v + bias.double())) <= 4e-6
    zz = z.double().requires_grad_(True)
    (dg,) = torch.autograd.grad(_gelu(zz).sum(), zz)
    assert rel(K.gemm(a, b, act=K.ACT_GELU_BWD, aux_in=z, **kw), v * dg) <= 4e-6
    assert rel(K.gemm(a, b, act=K.ACT_RELU_BWD, aux_in=z, residual=res, **kw), v * (z > 0) + res.double()) <= 4e-6
    strided = torch.full((m, n + 3), 5.0, device="cuda")
    K.gemm(a, b, out=strided[:, :n], residual=res, **kw)
    assert rel(strided[:, :n], v + res.double()) <= 2e-6 and bool((strided[:, n:] == 5.0).all())


def test_unaligned_operands():
    g = torch.Generator(device="cuda").manual_seed(1)
    buf = torch.randn(40 * 33 + 1, device="cuda", generator=g)
    a, b = buf[1:1 + 40 * 32].reshape(40, 32), torch.randn(24, 33, device="cuda", generator=g)[:, 1:]
    ref = a.double() @ b.double().t()
    assert float((K.gemm(a, b).double() - ref).norm() / ref.norm()) <= 2e-6


# A residual is [m, n], a row, a column or a scalar; the shapes beside them are refused, as are gradients of another shape.
@pytest.mark.parametrize("m,n,k", [(40, 24, 32), (70, 65, 16), (5, 1, 8), (1, 7, 8)])
def test_residual_shapes(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m + n)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    a, b, z = r(m, k), r(n, k), r(m, n)
    v = a.double() @ b.double().t()
    rel = lambda got, ref: float((got.double() - ref).norm() / ref.norm())
    for res in (r(n), r(1, n), r(m, 1), r(1), r(1, n).expand(m, n), r(n, m).t()):
        assert rel(K.gemm(a, b, residual=res), v + res.double()) <= 2e-6
        assert rel(K.gemm(a, b, act=K.ACT_RELU_BWD, aux_in=z, residual=res), v * (z > 0) + res.double()) <= 4e-6
    if m > 1 and n > 1:
        for res in (r(m - 1, n), r(m + 1, n), r(m, n + 1), r(1, m, n), r(2)):
            with pytest.raises(ValueError):
                K.gemm(a, b, residual=res)
        for aux in (r(m - 1, n), r(n), r(m, 1)):
            with pytest.raises(ValueError):
                K.gemm(a, b, act=K.ACT_GELU_BWD, aux_in=aux)
        with pytest.raises(RuntimeError):
            K.gemm(a, b, aux_out=torch.empty(m - 1, n, device="cuda"), act=K.ACT_GELU)
        with pytest.raises(RuntimeError):
            K.gemm(a, b, out=torch.empty(m - 1, n, device="cuda"), residual=z)


# Sliced reductions on two streams, and a captured one beside an eager one: each call's partial sums are its own.
@pytest.mark.parametrize("captured", [False, True])
def test_sliced_products_side_by_side(captured):
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    pairs = [(r(128, 4096), r(192, 4096)), (r(192, 2048), r(128, 2048))]
    alone = [K.gemm(*p) for p in pairs]                         # fixed order of slices: the same bits every time
    for (a, b), y in zip(pairs, alone):
        ref = a.double() @ b.double().t()
        assert float((y.double() - ref).norm() / ref.norm()) <= 2e-6
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = [[], []]
    graph = torch.cuda.CUDAGraph()
    if captured:
        with torch.cuda.graph(graph):
            replayed = K.gemm(*pairs[0])
    torch.cuda.synchronize()
    for _ in range(30):
        for i, st in enumerate(streams):
            with torch.cuda.stream(st):
                if captured and i == 0:
                    graph.replay()
                    outs[0].append(replayed.clone())
                else:
                    outs[i].append(K.gemm(*pairs[i]))
    torch.cuda.synchronize()
    for i in (0, 1):
        assert all(torch.equal(y, alone[i]) for y in outs[i])


# A residual or an activation gradient on top of a sliced reduction, and the time it may take: in one slice 128 x 128 x 4096 took
# eight times the plain product, with the epilogue in the kernel that adds the slices up it takes as long.
def test_sliced_epilogue():
    g = torch.Generator(device="cuda").manual_seed(5)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    rel = lambda got, ref: float((got.double() - ref).norm() / ref.norm())
    a, b, z, res, old = r(130, 4096), r(126, 4096), r(130, 126), r(130, 126), r(130, 126)
    v = a.double() @ b.double().t()
    assert rel(K.gemm(a, b, residual=res, alpha=0.5), 0.5 * v + res.double()) <= 2e-6
    assert rel(K.gemm(a, b, act=K.ACT_RELU_BWD, aux_in=z, residual=res), v * (z > 0) + res.double()) <= 4e-6
    aux = torch.empty(130, 126, device="cuda")
    y = K.gemm(a, b, act=K.ACT_GELU, aux_out=aux, out=old.clone(), accumulate=True)
    assert rel(aux, v) <= 2e-6 and rel(y, _gelu(v) + old.double()) <= 4e-6

    out = torch.empty(130, 126, device="cuda")
    assert graph_us(*[lambda: K.gemm(a, b, out=out, residual=res)] * 10) <= 2.5 * graph_us(*[lambda: K.gemm(a, b, out=out)] * 10)


# Ragged extents on an aligned pitch: the last 16-byte piece of a row or a column is copied in part.  What lies behind it is NaN, so a
# piece copied whole shows.  Tiles of 64 rows, of 32 rows, and a sliced reduction.
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k", [(70, 66, 17), (5, 3, 2), (33, 65, 130), (1001, 1000, 99), (1025, 903, 35), (90, 70, 514), (66, 62, 1027)])
def test_partial_vectors(m, n, k, a_mn, b_mn):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)

    def sliced(rows, cols):
        t = torch.full((rows, (cols + 3) // 4 * 4 + 4), float("nan"), device="cuda")
        t[:, :cols] = torch.randn(rows, cols, device="cuda", generator=g)
        return t[:, :cols]

    a, b = sliced(k, m) if a_mn else sliced(m, k), sliced(k, n) if b_mn else sliced(n, k)
    v = (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double()
    y = K.gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    assert float((y.double() - v).norm() / v.norm()) <= 2e-6
