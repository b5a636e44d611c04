"""Which operands the fp32 product's epilogue may address directly: everything else goes through the broadcasting sum, which refuses
what it cannot broadcast."""
import pytest
import torch

from oa_b200.ops import kernels as K


@pytest.mark.parametrize("shape,takes", [((5, 7), True), ((7,), False), ((1, 7), False), ((5, 1), False), ((1,), False), ((), False), ((4, 7), False),
                                         ((6, 7), False), ((5, 8), False), ((1, 5, 7), False)])
def test_epilogue_operand(shape, takes):
    assert K._f32_epilogue_takes(torch.zeros(shape), 5, 7) is takes


def test_epilogue_operand_layout():
    assert K._f32_epilogue_takes(None, 5, 7)
    assert K._f32_epilogue_takes(torch.zeros(5, 9)[:, 1:8], 5, 7)
    assert K._f32_epilogue_takes(torch.zeros(1, 7).expand(5, 7), 5, 7)
    assert not K._f32_epilogue_takes(torch.zeros(7, 5).t(), 5, 7)
    assert not K._f32_epilogue_takes(torch.zeros(5, 7, dtype=torch.bfloat16), 5, 7)


class _OnDevice:
    """What weight_grad looks at of a tensor on the device, with nothing behind it."""
    is_cuda, device = True, "cuda:0"

    def __init__(self, dtype, *shape):
        self.dtype, self.shape = dtype, shape

    def stride(self, i):
        return (self.shape[1], 1)[i]

    def numel(self):
        n = 1
        for d in self.shape:
            n *= d
        return n

    def is_contiguous(self):
        return True

    def data_ptr(self):
        return 0


@pytest.mark.parametrize("dtype,fused", [(torch.float32, True), (torch.bfloat16, False), (torch.float64, False)])
def test_weight_gradient_operands(dtype, fused, monkeypatch):
    # the kernel reads x as fp32: anything else belongs to gemm(), which refuses a mixture
    class Lib:
        def oa_gemm_f32_weight_grad(self, *a):
            went.append("fused")
            return 0

    went = []
    monkeypatch.setattr(K.N, "require", Lib)
    monkeypatch.setattr(K.N, "stream", lambda: 0)
    monkeypatch.setattr(K, "_f32_scratch", lambda *a: None)
    monkeypatch.setattr(K, "_launch", lambda *a, **k: None)
    monkeypatch.setattr(K, "gemm", lambda *a, **k: went.append("gemm"))
    monkeypatch.setattr(K, "col_sum", lambda *a, **k: went.append("col_sum"))
    f32 = lambda *s: _OnDevice(torch.float32, *s)
    K.weight_grad(f32(16, 8), _OnDevice(dtype, 16, 12), out=f32(8, 12), accumulate=False, bias_out=f32(8), bias_accumulate=False)
    assert went == (["fused"] if fused else ["gemm", "col_sum"])
