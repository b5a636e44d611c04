"""A decoding step that fails before its graph exists leaves the device-side position where it was."""
import pytest
import torch

from oa_b200.serve.decoder import _GraphedStep


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
