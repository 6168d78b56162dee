"""How many rows of logits the loss holds at a time."""
import pytest
import torch

from pisceslx_b200.ops.loss import rows_at_once


@pytest.mark.parametrize("T,V,H,rows", [
    (0, 1000, 64, 0), (1, 154856, 1024, 1), (2048, 154856, 4096, 2048),      # one chunk as before
    (2331, 154856, 1024, 2331), (8192, 32000, 4096, 8192),                   # no more than several chunks take, or than 2 GB
    (2730, 154856, 1024, 2730), (2731, 154856, 1024, 2048), (8192, 154856, 4096, 2048)])
def test_rows_at_once(T, V, H, rows):
    assert rows_at_once(T, V, H) == rows


@pytest.mark.parametrize("T,V,H", [(2331, 154856, 1024), (8192, 32000, 4096), (4700, 154856, 4096)])
def test_without_a_weight_gradient_there_is_no_sum_to_save(T, V, H):
    """Evaluation of 4700 rows over 154856 words: 2.9 GB of logits at once, 1.3 GB in chunks."""
    assert rows_at_once(T, V, H, weight_grad=False) == 2048 and rows_at_once(2000, V, H, weight_grad=False) == 2000


@pytest.mark.parametrize("grad,frozen,want", [(True, False, True), (True, True, False), (False, False, False)])
def test_the_model_says_whether_it_wants_the_weight_gradient(monkeypatch, grad, frozen, want):
    from pisceslx_b200 import YvConfig
    from pisceslx_b200.models import build_model, model as model_py
    cfg = YvConfig.tiny_text_moe()
    cfg.vocab_size, cfg.n_layer = 64, 1
    model = build_model(cfg, torch.device("cpu"), torch.float32)
    model.head_weight.requires_grad_(not frozen)
    seen = []
    monkeypatch.setattr(model_py, "rows_at_once", lambda *a, weight_grad=True: seen.append(weight_grad) or rows_at_once(*a))
    ids = torch.arange(12).view(2, 6)
    with torch.set_grad_enabled(grad):
        model(input_ids=ids, labels=ids)
    assert seen == [want]
