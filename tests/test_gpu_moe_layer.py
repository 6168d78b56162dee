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


@pytest.mark.parametrize("rows", [1, 64, 128, 512, 768, 1000])
def test_first_pass_of_a_recomputed_layer_equals_its_repetition(rows):
    """Recomputation runs the layer without a gradient first and with one later: the same function, bit for bit."""
    layer = _layer(2).train()
    layer.router.recomputing = True                 # leaves the routing statistics alone
    x = torch.randn(rows, layer.cfg.hidden_size, device=DEV).bfloat16()
    with torch.no_grad():
        first = layer(x)[0]
    again = layer(x)[0]
    assert again.requires_grad and torch.equal(first, again.detach())


@pytest.mark.parametrize("tokens", [40, 300])
def test_loss_and_gradients_do_not_depend_on_recomputation(tokens):
    from pisceslx_b200.models import build_model
    seen = []
    for recompute in (True, False):
        cfg = YvConfig.tiny_text_moe(vocab_size=512)
        cfg.n_layer, cfg.use_gradient_checkpointing = 2, recompute
        cfg.extra["moe_deterministic"] = True
        model = build_model(cfg, DEV, torch.bfloat16, seed=3).train()
        ids = torch.randint(0, 512, (2, tokens), device=DEV, generator=torch.Generator(DEV).manual_seed(1))
        loss = model(input_ids=ids, labels=ids, num_valid=2 * (tokens - 1))["loss"]
        loss.backward()
        seen.append([loss.detach()] + [layer.mlp.experts_w13.grad for layer in model.model.layers])
    assert all(torch.equal(a, b) for a, b in zip(*seen))


def test_gate_in_fp32_is_read_as_it_is():
    layer = _layer(1)
    layer.router.gate.float()
    x = torch.randn(9, layer.cfg.hidden_size, device=DEV).bfloat16()
    with torch.no_grad():
        layer.router(x)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured = layer.router(x)[0]
        layer.router.gate.weight.data.neg_()
        got, fresh = layer.router(x)[0], copy.deepcopy(layer.router)(x)[0]
        graph.replay()
    assert torch.equal(got, fresh) and torch.equal(captured, fresh)


@pytest.mark.parametrize("weights,period", [(0, 0), (3, 0), (12, 3), (5, 5), (3, -3), (0, 3)])
def test_row_weights_of_another_number_are_refused(weights, period):
    """One weight per row, or one per row modulo a period that divides the rows: the host checks it."""
    from pisceslx_b200.ops import kernels
    inp, dact = torch.zeros(12, 32, device=DEV).bfloat16(), torch.zeros(12, 16, device=DEV).bfloat16()
    out = (torch.empty_like(inp), torch.empty_like(dact), torch.empty(12, device=DEV))
    with pytest.raises(RuntimeError, match="swiglu_bwd_rows"):
        kernels().swiglu_bwd_rows(inp, dact, torch.ones(weights, device=DEV), *out, period)
