"""The model's token embedding with the options that ``nn.Embedding`` has."""
import pytest
import torch

from pisceslx_b200.models.model import YvTokenEmbedding


@pytest.mark.parametrize("option", [dict(), dict(padding_idx=2), dict(max_norm=0.5), dict(scale_grad_by_freq=True), dict(sparse=True)])
def test_options(option):
    torch.manual_seed(0)
    mine, plain = YvTokenEmbedding(7, 16, **option), torch.nn.Embedding(7, 16, **option)
    plain.load_state_dict(mine.state_dict())
    ids = torch.tensor([[1, 2, 2], [5, 1, 2]])
    out = []
    for m in (mine, plain):
        y = m(ids)
        (y * torch.arange(6.0).view(2, 3, 1)).sum().backward()
        out.append((y.detach(), m.weight.grad.to_dense(), m.weight.detach()))
    assert all(torch.equal(a, b) for a, b in zip(*out))
