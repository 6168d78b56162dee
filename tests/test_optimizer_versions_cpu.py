"""An optimizer's step is visible to whatever keeps a copy of a weight until the weight's version moves."""
import pytest
import torch
import torch.nn as nn

from pisceslx_b200.models.moe import YvSwiGLUExpert
from pisceslx_b200.optim.adamw import YvFusedAdamW
from pisceslx_b200.optim.ink import YvInkOptimizer
from pisceslx_b200.optim.muon import YvMuon
from pisceslx_b200.serve.fused_moe import PiscesLxFusedMoEDispatch

OPTIMIZERS = {
    "muon": lambda ps: YvMuon([(f"layer.{i}", p) for i, p in enumerate(ps)], lr=0.1),
    "adamw": lambda ps: YvFusedAdamW(ps, lr=0.1),
    "amsgrad": lambda ps: YvFusedAdamW(ps, lr=0.1, amsgrad=True),
    "ink": lambda ps: YvInkOptimizer(ps, lr=0.1),
}


@pytest.mark.parametrize("name", OPTIMIZERS)
def test_a_step_moves_the_versions_of_what_it_writes(name):
    torch.manual_seed(0)
    params = [nn.Parameter(torch.randn(s)) for s in ((8, 16), (16,), (2, 8, 8))]
    idle = nn.Parameter(torch.randn(4, 4))
    opt = OPTIMIZERS[name](params + [idle])
    for p in params:
        p.grad = torch.randn_like(p)
    before = [(p.detach().clone(), p._version) for p in params]
    version = idle._version
    opt.step()
    assert all(p._version > v and not torch.equal(p, old) for p, (old, v) in zip(params, before))
    assert idle._version == version


@pytest.mark.parametrize("name", OPTIMIZERS)
def test_stacked_experts_follow_a_step(name):
    torch.manual_seed(0)
    experts = nn.ModuleList([YvSwiGLUExpert(16, 32) for _ in range(4)])
    front, x = PiscesLxFusedMoEDispatch(4, 2), torch.randn(12, 16)
    weights, idx = torch.softmax(torch.randn(12, 4), -1).topk(2, -1)
    opt = OPTIMIZERS[name](list(experts.parameters()))
    with torch.no_grad():
        front(x, weights, idx, experts)
    for p in experts.parameters():
        p.grad = torch.randn_like(p)
    opt.step()
    with torch.no_grad():
        assert torch.equal(front(x, weights, idx, experts), PiscesLxFusedMoEDispatch(4, 2)(x, weights, idx, experts))
