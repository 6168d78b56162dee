"""A layer without a gradient works with its parameters as they are now, however they were written."""
import copy

import pytest
import torch

from pisceslx_b200 import YvConfig
from pisceslx_b200.models.moe_layer import YvDeepSeekMoELayer


def _layer(shared: int = 2) -> YvDeepSeekMoELayer:
    torch.manual_seed(0)
    cfg = YvConfig.tiny_text_moe(vocab_size=64)
    cfg.moe_shared_experts = shared
    layer = YvDeepSeekMoELayer(cfg)
    with torch.no_grad():
        for p in layer.parameters():
            p.normal_(0.0, 0.1)
    return layer


@pytest.mark.parametrize("training", [False, True])
def test_mixing_weights_written_through_data_are_used(training):
    layer = _layer().train(training)
    x = torch.randn(5, layer.cfg.hidden_size)
    with torch.no_grad():
        before = layer(x)[0]
        layer.shared_expert_weight.data.add_(torch.tensor([2.0, -2.0]))
        after, fresh = layer(x)[0], copy.deepcopy(layer)
        want = fresh(x)[0]
    assert torch.equal(after, want) and not torch.allclose(before, after, rtol=1e-3, atol=0)
