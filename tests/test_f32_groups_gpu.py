"""fp32 products whose blocks share the reduction out over groups of threads, and the kernel for short reductions beside them: reductions off
the stage of either, both sides of the line between them, rows on an aligned pitch, and the attention kernels on rows off 16 bytes."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


# Tiles for every SM (700 x 1400: 64-row tiles) and too few (200 x 132: 32-row tiles, below 512 columns of K in one piece); sums of up
# to 516 products of unit variance in any order: a few 2^-24 sqrt(K), below 2e-6 of the result's norm
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n", [(700, 1400), (200, 132), (31, 8)])
@pytest.mark.parametrize("k", [3, 28, 32, 36, 64, 184, 188, 192, 196, 260, 516])
def test_reductions(m, n, k, a_mn, b_mn):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    pitched = lambda rows, cols: torch.randn(rows, (cols + 7) // 4 * 4, device="cuda", generator=g)[:, :cols]
    a, b = pitched(k, m) if a_mn else pitched(m, k), pitched(k, n) if b_mn else pitched(n, k)
    ref = (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double()
    bias = torch.randn(n, device="cuda", generator=g)
    for got, want in ((K.gemm(a, b, a_mn=a_mn, b_mn=b_mn), ref), (K.gemm(a, b, a_mn=a_mn, b_mn=b_mn, bias=bias), ref + bias.double())):
        assert float((got.double() - want).norm() / want.norm()) <= 2e-6


@pytest.mark.parametrize("hd,off", [(32, 1), (32, 4), (64, 2), (64, 0)])
def test_attention_rows_off_16_bytes(hd, off):
    batch, seq, heads = 2, 70, 2
    D = heads * hd
    g = torch.Generator(device="cuda").manual_seed(hd + off)
    buf = torch.randn(batch * seq * 3 * D + 8, device="cuda", generator=g)
    qkv = buf[off:off + batch * seq * 3 * D].reshape(batch * seq, 3 * D)
    do = torch.randn(batch * seq, D, device="cuda", generator=g)
    parts = [qkv[:, i * D:(i + 1) * D] for i in range(3)]
    o, lse = K.flash_fwd(*parts, batch, seq, heads, hd)
    got = (o, *K.flash_bwd(*parts, o, do, lse, batch, seq, heads, hd))
    clean = [p.clone() for p in parts]
    o2, lse2 = K.flash_fwd(*clean, batch, seq, heads, hd)
    for a, e in zip(got, (o2, *K.flash_bwd(*clean, o2, do, lse2, batch, seq, heads, hd))):
        assert float((a - e).norm() / e.norm()) <= 1e-6       # the same sums but for the delta's, whose order follows the loads


# Weight and bias gradient from one product: in one piece, sliced, off the tile and with rows that the tile kernels do not take.
@pytest.mark.parametrize("rows,m,n", [(1, 4, 4), (37, 65, 12), (600, 70, 33), (2048, 128, 512), (2048, 512, 128), (500, 1000, 1400), (130, 700, 1500)])
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("off", [0, 1])
def test_weight_and_bias_gradient(rows, m, n, accumulate, off, monkeypatch):
    launch, names = K._launch, []
    monkeypatch.setattr(K, "_launch", lambda rc, name, *a, **k: (names.append(name), launch(rc, name, *a, **k)))
    g = torch.Generator(device="cuda").manual_seed(rows + m + n)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    dy, x = r(rows, (m + 7) // 4 * 4)[:, off:off + m], r(rows, (n + 3) // 4 * 4)[:, :n]
    w, b = r(m, n), r(m)
    want_w, want_b = dy.double().t() @ x.double(), dy.double().sum(0)
    if accumulate:
        want_w, want_b = want_w + w.double(), want_b + b.double()
    K.weight_grad(dy, x, out=w, accumulate=accumulate, bias_out=b, bias_accumulate=accumulate)
    # rows off 16 bytes take a product and a column sum of their own
    assert (names == ["oa_gemm_f32_weight_grad"]) if off == 0 else ("oa_gemm_f32_weight_grad" not in names and "oa_col_sum" in names), names
    assert float((w.double() - want_w).norm() / want_w.norm()) <= 2e-6
    # a column sum of up to 2048 terms of unit variance: a few 2^-24 times the partial sums it runs through, at most sqrt(rows) each
    assert float((b.double() - want_b).abs().max()) <= 2.0 ** -24 * 16 * (rows + 1) ** 0.5
    dy[0, 1] = float("inf")
    K.weight_grad(dy, x, out=w, accumulate=False, bias_out=b, bias_accumulate=False)
    assert float(b[1]) == float("inf") and bool(torch.isfinite(b[2:]).all())
