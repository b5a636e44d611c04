"""Projected rows of odd width: the chunked scan moves bf16 in pairs, so such rows go through the sequential kernels, and its entry
points answer OA_ERR_ALIGN before they launch anything."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

from oa_b200 import _native as N
from oa_b200.ops import kernels as K
from oa_b200.ops import mamba3 as M3


@pytest.mark.parametrize("heads,angles,at,chunked", [(1, 32, 0, False), (2, 32, 0, True), (3, 16, 0, False), (1, 33, 0, True), (2, 32, 2, False), (2, 32, 4, True)])
def test_route(heads, angles, at, chunked, monkeypatch):
    monkeypatch.delenv("OA_MAMBA3_SSD", raising=False)
    monkeypatch.delenv("OA_MAMBA3_SSD_FUSED", raising=False)
    d = M3.Mamba3Dims(heads * 64, heads, 64, 128, angles)
    proj = SimpleNamespace(is_cuda=True, dtype=torch.bfloat16, data_ptr=lambda: 0x10000 + at)
    assert M3._use_ssd(proj, d, 256) is chunked
    monkeypatch.setenv("OA_MAMBA3_SSD_FUSED", "0")
    assert M3._use_ssd(proj, d, 256)                 # the statement of the chunked form indexes single columns


BASE, B, L, H, P = 0x10000, 1, 128, 1, 64


def _entry(name, *args):
    path = N.lib_path()
    if not path.exists():
        pytest.skip("kernel library not built")
    f = getattr(ctypes.CDLL(str(path)), name)
    f.restype, f.argtypes = next((r, a) for n, r, a in N._PROTOS if n == name)
    return f(*args, None)


# one operand at a time off its boundary; addresses that nothing may touch
@pytest.mark.parametrize("x,ldx,bb", [(BASE, 387, BASE), (BASE + 2, 388, BASE), (BASE, 388, BASE + 4)])
def test_prep_fwd(x, ldx, bb):
    assert _entry("oa_ssd_prep_fwd", x, ldx, BASE, BASE, bb, *[BASE] * 15, B, L, H, P, 128, 32) == N.CONST["OA_ERR_ALIGN"]


@pytest.mark.parametrize("z,ldz,y,yraw,ldy", [(BASE, 387, BASE, BASE, 64), (BASE + 2, 388, BASE, BASE, 64), (BASE, 388, BASE + 2, BASE, 64),
                                              (BASE, 388, BASE, BASE + 2, 64), (None, 0, BASE, None, 65)])
def test_out_fwd(z, ldz, y, yraw, ldy):
    assert _entry("oa_ssd_out_fwd", BASE, z, ldz, y, yraw, ldy, B, L, H, P) == N.CONST["OA_ERR_ALIGN"]


@pytest.mark.parametrize("dy,ldy,z,ldz,dz,lddz", [(BASE + 2, 64, None, 0, None, 0), (BASE, 65, None, 0, None, 0), (BASE, 64, BASE, 387, BASE, 388),
                                                  (BASE, 64, BASE, 388, BASE, 387), (BASE, 64, BASE, 388, BASE + 2, 388)])
def test_dy_prep(dy, ldy, z, ldz, dz, lddz):
    assert _entry("oa_ssd_dy_prep", dy, BASE if z else None, ldy, z, ldz, dz, lddz, BASE, B, L, H, P) == N.CONST["OA_ERR_ALIGN"]


@pytest.mark.parametrize("dx,lddx", [(BASE, 387), (BASE + 2, 388)])
def test_dx_out(dx, lddx):
    assert _entry("oa_ssd_dx_out", BASE, BASE, BASE, BASE, dx, lddx, BASE, B, L, H, P) == N.CONST["OA_ERR_ALIGN"]


# One head per call, as a layer with a B and C projection per head makes them (3 + 32 scalar columns), and biases that start anywhere.
@pytest.mark.gpu
@pytest.mark.parametrize("H,A,has_z", [(1, 32, True), (3, 16, False), (2, 16, True)])
def test_core(H, A, has_z):
    P, Nn, L = 64, 128, 256
    d = M3.Mamba3Dims(H * P, H, P, Nn, A, has_z=has_z)
    g = torch.Generator().manual_seed(H + A)
    r = lambda *s: torch.randn(*s, generator=g)
    proj, dy = r(L, d.d_in_proj).bfloat16(), r(L, d.d_inner).bfloat16()
    proj[:, 2 * d.d_inner + 2 * Nn:] *= 0.5
    params = (0.5 * r(1, H) - 3.0, 1 + 0.1 * r(H, Nn), 1 + 0.1 * r(H, Nn), r(H))
    off = lambda t: torch.cat((torch.zeros(1), t.flatten())).cuda()[1:].view(t.shape)
    y, s = M3.core_fwd(proj.cuda(), *map(off, params), d, 1, L)
    assert (s.ssd is None) == bool(d.d_in_proj % 2)
    dy_off = torch.cat((torch.zeros(1).bfloat16(), dy.flatten())).cuda()[1:].view(dy.shape)
    got = M3.core_bwd(s, dy_off)
    torch.cuda.synchronize()
    K.check_status()
    yr, sr = M3.core_fwd(proj.float(), *params, d, 1, L)
    ref = M3.core_bwd(sr, dy.float())
    rel = lambda a, e: float((a.double().cpu() - e.double()).norm() / e.double().norm())
    # as for the fused chunk kernels: bf16 operands of long fp32 sums, and sums over all rows that cancel
    assert rel(y, yr) <= 1e-2
    z = 0 if has_z else d.d_inner
    assert rel(got[0][:, z:], ref[0][:, z:]) <= 2e-2
    for a, e in zip(got[1:], ref[1:]):
        assert rel(a.view(e.shape), e) <= 4e-2
