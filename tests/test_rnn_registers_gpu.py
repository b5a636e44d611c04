"""Recurrent scans with the weights in registers: hidden widths at the edges of the 16-wide pieces, odd batches, initial state."""
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gates", [1, 3])
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-5), (torch.bfloat16, 4e-2)])
@pytest.mark.parametrize("B,S,H", [(1, 1, 8), (3, 2, 24), (2, 5, 32), (5, 9, 40), (2, 33, 64), (3, 6, 72), (2, 17, 128), (150, 4, 128), (2, 4, 136), (2, 4, 20)])
def test_scan(gates, dtype, tol, B, S, H):
    g = torch.Generator().manual_seed(B * 1009 + S * 31 + H)
    r = lambda *s, k=1.0: (k * torch.randn(*s, generator=g)).to(dtype)
    gi, w, b, h0, do = r(B, S, gates * H), r(gates * H, H, k=H ** -0.5), r(gates * H, k=0.1), r(B, H, k=0.5), r(B, S, H)
    c = lambda t: t.float()
    for bias in (b, None):
        cb = c(bias) if bias is not None else None
        gb = bias.cuda() if bias is not None else None
        out, hp = K.rnn_scan_fwd(gi.cuda(), w.cuda(), gb, gates, h0=h0.cuda())
        outr, hpr = K.rnn_scan_fwd(c(gi), c(w), cb, gates, h0=c(h0))
        assert (out.float().cpu() - outr).abs().max().item() <= tol
        assert (hp.float().cpu() - hpr).abs().max().item() <= tol
        got = K.rnn_scan_bwd(gi.cuda(), w.cuda(), gb, hpr.to(dtype).cuda(), do.cuda(), gates)
        ref = K.rnn_scan_bwd(c(gi), c(w), cb, hpr.to(dtype).float(), c(do), gates)
        for a, e, nm in zip(got, ref, ("dgi", "dgh", "dh0")):
            assert (a.float().cpu() - e).abs().max().item() <= tol * max(1.0, e.abs().max().item()), nm
    torch.cuda.synchronize()


# The coefficients that the forward scan leaves: the same gradients as from the scan that works them out again.
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-5), (torch.bfloat16, 4e-2)])
@pytest.mark.parametrize("B,S,H", [(1, 1, 80), (3, 2, 96), (2, 33, 112), (150, 5, 128), (2, 64, 128), (2, 5, 72)])
def test_forward_coefficients(dtype, tol, B, S, H):
    g = torch.Generator().manual_seed(B * 1009 + S * 31 + H)
    r = lambda *s, k=1.0: (k * torch.randn(*s, generator=g)).to(dtype)
    gi, w, b, h0, do = r(B, S, 3 * H), r(3 * H, H, k=H ** -0.5), r(3 * H, k=0.1), r(B, H, k=0.5), r(B, S, H)
    coef = K.rnn_coef(gi.cuda(), 3)
    assert (coef is None) == (H % 16 != 0)
    if coef is not None:
        coef.fill_(float("nan"))
    out, hp = K.rnn_scan_fwd(gi.cuda(), w.cuda(), b.cuda(), 3, h0=h0.cuda(), coef=coef)
    got = K.rnn_scan_bwd(gi.cuda(), w.cuda(), b.cuda(), hp, do.cuda(), 3, coef=coef)
    outr, hpr = K.rnn_scan_fwd(gi.float(), w.float(), b.float(), 3, h0=h0.float())
    ref = K.rnn_scan_bwd(gi.float(), w.float(), b.float(), hpr, do.float(), 3)
    assert (out.float().cpu() - outr).abs().max().item() <= tol
    for a, e, nm in zip(got, ref, ("dgi", "dgh", "dh0")):
        assert (a.float().cpu() - e).abs().max().item() <= tol * max(1.0, e.abs().max().item()), nm


def test_coefficients_held_are_bounded(monkeypatch):
    # four scans on one tape, room for the coefficients of two: the others' backward scans work theirs out again, with the same gradients
    from oa_b200.core.matrix import OaMatrix
    from oa_b200.ml import autograd as AG
    from oa_b200.ml.nn.recurrent import RecurrentScan

    B, S, H = 4, 96, 128
    share = 4 * K.rnn_coef(torch.empty(B, S, 3 * H, device="cuda"), 3).numel()
    monkeypatch.setattr(AG, "KEEP_BYTES", 2 * share + share // 2)
    g = torch.Generator(device="cuda").manual_seed(5)
    w, b = torch.randn(3 * H, H, device="cuda", generator=g) * H ** -0.5, torch.randn(3 * H, device="cuda", generator=g) * 0.1
    x, do = torch.randn(B, S, 3 * H, device="cuda", generator=g), torch.randn(B, S, H, device="cuda", generator=g)

    def scans():
        xs = [OaMatrix(x.clone()) for _ in range(4)]
        ws = [OaMatrix(w.clone()) for _ in range(4)]
        for m in xs + ws:
            m.SetRequiresGrad(True)
        return xs, ws

    for _ in range(2):                                          # the share comes back with the backward pass
        xs, ws = scans()
        with AG.OaGradientTape() as tape:
            torch.cuda.synchronize()
            before = torch.cuda.memory_allocated()
            outs = [RecurrentScan(m, v, OaMatrix(b), 3, "GruScan") for m, v in zip(xs, ws)]
            held = torch.cuda.memory_allocated() - before
            assert held <= 4 * 2 * (4 * B * S * H) + 2 * share + 8 * 512        # outputs, previous states, two scans' coefficients
            for o in outs:
                tape.Backward(o, do)
            assert AG.Keeping().left == AG.KEEP_BYTES
    dx = [m.GradTensor() for m in xs]
    dw = [m.GradTensor() for m in ws]
    for i in (1, 2, 3):                                         # each within the 2e-5 of the tests above
        assert float((dx[i] - dx[0]).abs().max()) <= 4e-5 * max(1.0, float(dx[0].abs().max()))
        assert float((dw[i] - dw[0]).norm()) <= 4e-5 * float(dw[0].norm())
