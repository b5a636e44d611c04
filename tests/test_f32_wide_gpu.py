"""fp32 products whose tiles fit one wave of blocks, and those whose slices of K a cluster adds up, against 64 bits and against the general kernel."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu

TOL = 2e-6          # sums of at most 3000 products of unit variance in any order: a few 2^-24 sqrt(K) of the result's norm


def _rel(got, want):
    return float((got.double() - want).norm() / want.norm())


# 32-row tiles for exactly the chip and one more, 64-row tiles likewise; clusters of eight, four and two, with slices off four columns; the sizes around each line; eight
# columns of K and nine
SHAPES = [(1, 1, 4), (148 * 32, 64, 40), (148 * 32 + 1, 60, 40), (148 * 64, 64, 33), (148 * 64 + 1, 64, 33), (130, 130, 300),
          (20, 48, 8), (20, 48, 9), (2048, 130, 5), (128, 128, 513), (100, 190, 1021), (65, 385, 1024), (512, 128, 1537), (512, 130, 3000), (64, 1024, 700), (33, 2048, 1536)]


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_epilogues(m, n, k, a_mn, b_mn):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    r = lambda rows, cols, off=0: torch.randn(rows, (cols + 7) // 4 * 4, device="cuda", generator=g)[:, off:off + cols]
    a, b = r(k, m) if a_mn else r(m, k), r(k, n) if b_mn else r(n, k)
    want = 0.5 * ((a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double())
    bias = torch.randn(n, device="cuda", generator=g)
    for off in (0, 1):                    # rows of the result on 16 bytes and off
        res, out, aux = r(m, n, off), r(m, n, off), r(m, n, off)
        before = out.double()
        got = K.gemm(a, b, a_mn=a_mn, b_mn=b_mn, alpha=0.5, bias=bias, residual=res, out=out, accumulate=True, act=K.ACT_RELU, aux_out=aux)
        z = want + bias.double()
        assert _rel(aux, z) <= TOL
        assert _rel(got, torch.relu(z) + res.double() + before) <= TOL
    pad = lambda t: torch.cat([t.new_zeros(t.shape[0], 1), t], 1)[:, 1:]      # off 16 bytes: the general kernel
    assert _rel(K.gemm(a, b, a_mn=a_mn, b_mn=b_mn, alpha=0.5), K.gemm(pad(a), pad(b), a_mn=a_mn, b_mn=b_mn, alpha=0.5).double()) <= TOL


@pytest.mark.parametrize("rows,m,n", [(512, 128, 128), (1030, 100, 128), (2048, 512, 128), (1500, 128, 384), (1028, 384, 256), (77, 300, 300)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_weight_and_bias_gradient(rows, m, n, accumulate):
    g = torch.Generator(device="cuda").manual_seed(rows + m)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    dy, x, w, b = r(rows, m), r(rows, n), r(m, n), r(m)
    want_w, want_b = dy.double().t() @ x.double(), dy.double().sum(0)
    if accumulate:
        want_w, want_b = want_w + w.double(), want_b + b.double()
    first = K.weight_grad(dy, x, out=w.clone(), accumulate=accumulate, bias_out=b.clone(), bias_accumulate=accumulate)
    K.weight_grad(dy, x, out=w, accumulate=accumulate, bias_out=b, bias_accumulate=accumulate)
    assert _rel(w, want_w) <= TOL and _rel(b, want_b) <= TOL
    assert first is None or torch.equal(first[0] if isinstance(first, tuple) else first, w)      # the same order every time


def test_batch_in_one_wave():
    g = torch.Generator(device="cuda").manual_seed(3)
    a, b = torch.randn(5, 70, 36, device="cuda", generator=g), torch.randn(5, 36, 52, device="cuda", generator=g)
    assert _rel(K.bmm_f32(a, b, b_mn=True), a.double() @ b.double()) <= TOL
