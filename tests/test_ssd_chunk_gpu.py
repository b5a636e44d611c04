"""The fused chunk kernels of the Mamba-3 scan (state width 128, head width 64) against the plain statement of the chunked form."""
import pytest
import torch

from oa_b200.ops import kernels as K
from oa_b200.ops import mamba3 as M3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("has_z", [False, True])
# the last three have one to two, two to three and three to four chunks to each of 148 CTAs, so that the backward kernel's regions and barriers come round
@pytest.mark.parametrize("B,L,H,A,skip", [(1, 128, 1, 32, True), (2, 256, 3, 16, False), (1, 640, 2, 0, True), (2, 384, 40, 32, True), (2, 640, 40, 16, True),
                                          (1, 1536, 40, 32, False)])
def test_chunk_scan(B, L, H, A, skip, has_z):
    P, N = 64, 128
    g = torch.Generator().manual_seed(L + H + A)
    pad = (-(3 * H + A)) % 8
    d = M3.Mamba3Dims(H * P, H, P, N, A + pad if A else 0, has_z=has_z)
    if d.angles == 0 and d.d_in_proj % 8:
        d = M3.Mamba3Dims(H * P, H, P, N, 8, has_z=has_z)
    if d.d_in_proj % 8:
        d.angles += (-d.d_in_proj) % 8
    rows = B * L
    proj = torch.randn(rows, d.d_in_proj, generator=g).bfloat16()
    dtb, Bb, Cb = 0.5 * torch.randn(1, H, generator=g) - 3.0, 1 + 0.1 * torch.randn(H, N, generator=g), 1 + 0.1 * torch.randn(H, N, generator=g)
    D = torch.randn(H, generator=g) if skip else None
    dy = torch.randn(rows, d.d_inner, generator=g).bfloat16()
    c = lambda t: None if t is None else t.cuda()
    y, s = M3.core_fwd(c(proj), c(dtb), c(Bb), c(Cb), c(D), d, B, L)
    assert s.ssd.M is None                                      # the fused path
    got = M3.core_bwd(s, c(dy))
    torch.cuda.synchronize()
    K.check_status()
    yr, sr = M3.core_fwd(proj.float(), dtb, Bb, Cb, D, d, B, L)
    ref = M3.core_bwd(sr, dy.float())
    rel = lambda a, e: float((a.double().cpu() - e.double()).norm() / e.double().norm().clamp_min(1e-9))
    # bf16 operands of 128-long fp32 sums: a few roundings of 2^-9 each; sums over all rows cancel and keep up to four times that
    assert rel(y, yr) <= 1e-2
    o = d.offsets()
    for nm, lo, hi in (("z", o[0], o[1]), ("x", o[1], o[2]), ("B", o[2], o[3]), ("C", o[3], o[4]), ("dt", o[4], o[5]), ("a", o[5], o[6]),
                       ("trap", o[6], o[7]), ("angle", o[7], d.d_in_proj)):
        if hi > lo and (nm != "z" or has_z):
            assert rel(got[0][:, lo:hi], ref[0][:, lo:hi]) <= 2e-2, nm
    for nm, a, e in zip(("dt_bias", "B_bias", "C_bias", "D"), got[1:], ref[1:]):
        if e is not None:
            assert rel(a, e) <= 4e-2, nm


@pytest.mark.parametrize("what", ["infinite row", "fast decay"])
def test_later_tokens_are_chosen_away(what):
    """A token's scores with later ones are not part of anything, whatever they hold: a C that is infinite in one token (its own scores with all
    others are NaN), and decays so fast that the factor towards later tokens overflows."""
    B, L, H, P, N = 1, 512, 75, 64, 128                         # 300 chunks
    d = M3.Mamba3Dims(H * P, H, P, N, 16 + (-(3 * H + 16)) % 8)
    assert d.d_in_proj % 8 == 0
    g = torch.Generator(device="cuda").manual_seed(5)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    proj, dy, o = r(L, d.d_in_proj).bfloat16(), r(L, d.d_inner).bfloat16(), d.offsets()
    dtb, Bb, Cb = torch.full((1, H), 4.0 if what == "fast decay" else -3.0, device="cuda"), 1 + 0.1 * r(H, N), 1 + 0.1 * r(H, N)

    def run(p):
        y, s = M3.core_fwd(p, dtb, Bb, Cb, None, d, B, L)
        assert s.ssd.M is None
        return y.clone(), M3.core_bwd(s, dy)[0][:, o[1]:o[2]].clone()

    y, dx = run(proj)
    assert bool(y.isfinite().all()) and bool(dx.isfinite().all())
    if what == "infinite row":
        at = 200                                                # inside a chunk, in its second 32 rows
        proj[at, o[3]:o[4]] = float("inf")
        y2, dx2 = run(proj)
        others = torch.arange(L, device="cuda") != at
        assert torch.equal(y2[others], y[others]) and not bool(y2[at].isfinite().any())
        assert torch.equal(dx2[at + 1:], dx[at + 1:])           # what a later token gives is none of this one's business
    torch.cuda.synchronize()
    K.check_status()
