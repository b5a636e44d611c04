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
