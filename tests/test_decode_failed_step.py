"""Decoding steps at the edges: one that fails before its graph exists leaves the device-side position where it was; models without blocks."""
import pytest
import torch

from oa_b200.models import OaGptConfig, OaGptModel
from oa_b200.serve.decoder import OaGptDecoder, _GraphedStep


def test_position_after_a_failed_first_step():
    g = _GraphedStep(torch.device("cpu"), 2)
    g.pos.fill_(6)

    def fails(ids):
        raise RuntimeError("no room")

    for _ in range(2):
        with pytest.raises(RuntimeError, match="no room"):
            g.run(torch.zeros(2, 1, dtype=torch.int32), fails, begin=lambda ids: g.pos.add_(1))
        assert g.pos.item() == 6 and g.graph is None


def test_position_when_the_step_itself_counts():
    """Without work in front of the graph the captured function adds one at its end, which a failure does not reach."""
    g = _GraphedStep(torch.device("cpu"), 2)

    def fails(ids):
        raise RuntimeError("no room")

    with pytest.raises(RuntimeError, match="no room"):
        g.run(torch.zeros(2, 1, dtype=torch.int32), fails)
    assert g.pos.item() == 0


def test_a_model_without_blocks_takes_the_general_step():
    model = OaGptModel(OaGptConfig(64, 32, 0, 4, 64, 32, "rms", "swiglu", 10000.0, False, 1e-5, 0.3))
    dec = OaGptDecoder(model, 2, 8)
    assert not dec._fusable()                          # the joined step begins with the first block's norm
    assert dec.Step(torch.zeros(2, 1, dtype=torch.int32)).shape == (2, 64)
