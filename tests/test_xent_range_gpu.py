"""Cross-entropy of rows far from zero: whole rows, single peaks and masks of every size, in each kernel that the launch chooses between."""
import numpy as np
import pytest
import torch

from oa_b200.ops import kernels as K

pytestmark = pytest.mark.gpu

SIZES = [1e4, 1e6, 1e9, 1e10, 1e12, 1e20, 1e30, 3e38]
# one warp per row; a row on the chip with 128, 256 and 512 threads, with a remainder off the vectors; the online kernel (rows off 16 bytes)
KERNELS = [(512, 0), (4096, 0), (4100, 0), (8000, 0), (16200, 0), (32008, 0), (20003, 0), (4096, 1)]


def _rows(vocab, dtype, rows, off):
    g = torch.Generator(device="cuda").manual_seed(vocab + off)
    ld = (vocab + off + 7) // 8 * 8
    x = torch.zeros(len(rows), ld, device="cuda")
    for i, (kind, c) in enumerate(rows):
        r = torch.randn(vocab, device="cuda", generator=g) * 2
        if kind == "whole":
            r[:] = c
        elif kind == "peak":
            r[vocab // 3] = c
        elif kind == "masked":                             # a thread's first vectors hold nothing else, and some threads' all of them
            r[:vocab // 2] = c
        elif kind == "all but one":
            r[:vocab - 1] = c
        else:
            r += c
        x[i, off:off + vocab] = r
    return x.to(dtype)[:, off:off + vocab]


def _run(x, t, ignore=-100):
    d = torch.zeros(x.shape[0], x.stride(0), dtype=x.dtype, device="cuda")
    off = x.storage_offset()
    return K.xent_fwd_bwd(x, t, grad_scale=0.5, ignore_index=ignore, dlogits=d[:, off:off + x.shape[1]])


def _reference(x, t):
    """In 64 bits, but for the log-sum-exp that fp32 holds: far from zero its rounding is most of a result's error, and log(vocab) is lost."""
    r = x.double()
    exact = torch.logsumexp(r, 1)
    lse = exact.float().double()
    p = torch.exp(r - lse[:, None])
    p[torch.arange(len(t)), t.long()] -= 1.0
    ulp = torch.from_numpy(np.spacing(np.abs(lse.float().cpu().numpy()))).double().cuda()
    return exact, lse - r.gather(1, t.long()[:, None])[:, 0], 0.5 * p, ulp


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("vocab,off", KERNELS)
def test_rows_of_any_size(vocab, off, dtype):
    rows = [("whole", s * c) for c in SIZES for s in (1, -1)] + [("peak", c) for c in SIZES]
    rows += [(kind, c) for kind in ("masked", "all but one") for c in [-c for c in SIZES] + [float("-inf")]]
    x = _rows(vocab, dtype, rows, off)
    t = torch.full((len(rows),), vocab - 1, device="cuda", dtype=torch.int32)       # a logit that no mask and no peak covers
    loss, d = _run(x, t)
    _, ref, grad, ulp = _reference(x, t)
    # a sum near a tie may round the other way: one unit in the last place of the log-sum-exp, which is a factor on the probabilities
    # (a unit of many counts as two results that cannot both be told apart: 0 or 1).  Beside it 2e-6 of exponentials and sums.
    tol = ulp + 2e-6
    assert bool(((loss.double() - ref).abs() <= tol * (1 + ref.abs())).all()), (rows, loss, ref)
    err, size = (d.double() - grad).norm(dim=1), 0.5 + grad.norm(dim=1)      # the target's entry is the difference of two numbers of up to 1/2
    tol = torch.where(ulp < 0.1, tol, torch.full_like(tol, 1e-6)) + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
    assert bool((err <= tol * size).all()), [(r, float(a), float(b)) for r, a, b in zip(rows, err, tol * size) if not a <= b]
    # rows that do not count
    loss, d = _run(x, t, ignore=vocab - 1)
    assert bool((loss == 0).all()) and bool((d == 0).all())


@pytest.mark.parametrize("vocab,off", KERNELS)
@pytest.mark.parametrize("shift", [0.0, 30.0, -30.0, 100.0, 1e3, -1e4, 1e4])
def test_error_of_ordinary_rows(vocab, off, shift):
    """fp32 rows beside zero and away from it: no more than half a unit of the log-sum-exp, and the exponentials' own 1e-6."""
    x = _rows(vocab, torch.float32, [("shifted", shift)] * 24, off)
    t = torch.arange(24, device="cuda", dtype=torch.int32) * (vocab // 24)
    loss, d = _run(x, t)
    exact, _, _, ulp = _reference(x, t)
    r = x.double()
    grad = torch.exp(r - exact[:, None])
    grad[torch.arange(24), t.long()] -= 1.0
    grad *= 0.5
    other = torch.ones_like(grad, dtype=torch.bool)
    other[torch.arange(24), t.long()] = False              # the target's entry is about -1 and hides the rest in a norm
    e, g = ((d.double() - grad) * other).norm(dim=1), (grad * other).norm(dim=1)
    assert bool((e <= (0.5 * ulp + 1e-6) * g).all()), (e / g, ulp)
    want = exact - r.gather(1, t.long()[:, None])[:, 0]
    assert bool(((loss.double() - want).abs() <= ulp + 1e-6 * want.abs().clamp_min(1.0)).all())
