"""The mixture-of-experts layer on the GPU: what it derives from its parameters, and its passes with and without a gradient."""
import copy

import pytest
import torch

from pisceslx_b200 import YvConfig
from pisceslx_b200.models.moe_layer import YvDeepSeekMoELayer
from pisceslx_b200.ops import functional as F_

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _layer(shared: int, mix_dtype: torch.dtype = torch.bfloat16) -> YvDeepSeekMoELayer:
    torch.manual_seed(0)
    cfg = YvConfig.tiny_text_moe(vocab_size=64)
    cfg.moe_shared_experts = shared
    cfg.extra["moe_deterministic"] = True
    layer = YvDeepSeekMoELayer(cfg).to(DEV, torch.bfloat16)
    layer.router.expert_bias.data = layer.router.expert_bias.data.float()
    with torch.no_grad():
        for p in layer.parameters():
            p.normal_(0.0, 0.1)
        layer.shared_expert_weight.data = layer.shared_expert_weight.data.to(mix_dtype)
    return layer.eval()


@pytest.mark.parametrize("shared,dtype", [(1, torch.bfloat16), (2, torch.float32), (5, torch.bfloat16)])
@pytest.mark.parametrize("rows", [1, 128, 129])
def test_mixing_weights_are_read_from_the_parameter(rows, shared, dtype):
    """Inside the few-row product and beside it; after a write that leaves no trace in the parameter's version, and by a
    captured pass."""
    layer = _layer(shared, dtype)
    x = torch.randn(rows, layer.cfg.hidden_size, device=DEV).bfloat16()
    with torch.no_grad():
        layer._shared(x)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured = layer._shared(x)
        layer.shared_expert_weight.data.copy_(torch.linspace(-3.0, 2.0, shared, device=DEV))
        got, fresh = layer._shared(x), copy.deepcopy(layer)._shared(x)
        graph.replay()
        assert torch.equal(got, fresh) and torch.equal(captured, fresh)
        S, Fs, d = shared, layer.shared_ffn, torch.float64
        gate, up = (x.to(d) @ layer.shared_w13.to(d).t()).view(rows, S, 2, Fs).unbind(2)
        act = torch.nn.functional.silu(gate) * up * torch.softmax(layer.shared_expert_weight.to(d), 0)[:, None]
        want = act.reshape(rows, S * Fs) @ layer.shared_w2.to(d).t()
    # the products, the activation and the result are rounded to bf16, 2^-9 of a value each
    assert (got.double() - want).norm() < 3 * 2.0 ** -8 * want.norm()


@pytest.mark.parametrize("parts", [1, 3])
def test_softmax_inside_the_product(parts):
    g = torch.Generator(DEV).manual_seed(parts)
    x = torch.randn(33, 256, device=DEV, generator=g).bfloat16()
    w = (torch.randn(parts * 128, 256, device=DEV, generator=g) / 16).bfloat16()
    logits = torch.randn(parts, device=DEV, generator=g) * 4
    inside = F_.skinny_swiglu(x, w, 64, logits, True)
    factors = F_.skinny_swiglu(x, w, 64, torch.softmax(logits, 0))
    # the factors differ by a few roundings in fp32, which move a bf16 result to its neighbour at most
    assert (inside.float() - factors.float()).abs().max() <= 2.0 ** -7 * factors.float().abs().max()
    assert (inside.double() - factors.double()).norm() < 2.0 ** -12 * factors.double().norm()
