"""Gradients of attention whose bits repeat: those of the kernels with one writer for every row, which torch's switch selects, by the
argument and by the models' option."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _reference(grads):
    torch.use_deterministic_algorithms(True)
    try:
        return grads()
    finally:
        torch.use_deterministic_algorithms(False)


def _same(a, b):
    assert len(a) == len(b) and all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
def test_argument(d, causal):
    from pisceslx_b200.ops import functional as F_
    from pisceslx_b200.ops.reference import rope_tables
    from pisceslx_b200.parallel.cp import _block_backward
    g = torch.Generator("cuda").manual_seed(d)
    S, hq, hk = 1900, 4, 2
    rand = lambda w: torch.randn(S, w * d, device="cuda", generator=g).to(BF16)
    q, k, v, do = (rand(h).requires_grad_(True) for h in (hq, hk, hk, hq))
    qkv = torch.cat([q, k, v], 1).detach().requires_grad_(True)
    cu = torch.tensor([0, S], dtype=torch.int32, device="cuda")
    pos = torch.arange(S, dtype=torch.int32, device="cuda")
    cos, sin = rope_tables(S, d, 1e4, device="cuda")

    def separate(**more):
        return torch.autograd.grad(F_.attention(q, k, v, cu, None, S, S, hq, hk, d, causal, **more), (q, k, v), do)

    def fused(**more):
        return torch.autograd.grad(F_.rope_attention(qkv.clone(), cos, sin, pos, cu, S, hq, hk, d, d, causal, **more), qkv, do)

    def block(**more):
        o, lse = torch.empty_like(q), torch.empty(hq, S, device="cuda")
        from pisceslx_b200.ops import kernels, status_word
        kernels().attn_fwd(q, k, v, o, lse, cu, None, S, S, hq, hk, d, causal, d ** -0.5, status_word(q.device))
        return _block_backward(do, q, k, v, o, lse, hq, hk, d, causal, d ** -0.5, **more)

    for grads in (separate, fused, block):
        want = _reference(grads)
        for _ in range(3):
            _same(grads(deterministic=True), want)


def test_option_of_the_models():
    """Every gradient of a text layer's attention and of a block of the vision encoder."""
    from pisceslx_b200 import YvConfig
    from pisceslx_b200.models.attention import AttnContext, YvAttention
    from pisceslx_b200.models.multimodal import YvVisionEncoder
    from pisceslx_b200.ops.reference import rope_tables
    torch.manual_seed(0)
    cfg = YvConfig.tiny_text_moe()
    cfg.extra["moe_deterministic"] = True
    layer = YvAttention(cfg, 0).to("cuda", BF16)
    S = 1500
    x = torch.randn(S, cfg.hidden_size, device="cuda").to(BF16)
    cu = torch.tensor([0, S], dtype=torch.int32, device="cuda")
    cos, sin = rope_tables(S, layer.rot_dim, 1e4, device="cuda")
    ctx = AttnContext(cos=cos, sin=sin, positions=torch.arange(S, dtype=torch.int32, device="cuda"), cu_seqlens=cu, max_len=S)
    seed = torch.randn(S, cfg.hidden_size, device="cuda").to(BF16)
    text = lambda: torch.autograd.grad(layer(x, ctx), list(layer.parameters()), seed)
    encoder = YvVisionEncoder(cfg, dim=256, depth=1, heads=4).to("cuda", BF16)
    y, grad = (torch.randn(S, 256, device="cuda").to(BF16) for _ in range(2))
    vision = lambda: torch.autograd.grad(encoder.blocks[0](y, cu, S), list(encoder.blocks[0].parameters()), grad)
    for grads in (text, vision):
        want = _reference(grads)
        for _ in range(3):
            _same(grads(), want)


def test_scratch_of_the_backward_is_bounded():
    """Sums of one KV head above the bound (300 000 tokens of 8 query heads of 64: 614 MB): the two kernels."""
    from pisceslx_b200.ops import functional as F_
    T, hq, hk, d, S = 300000, 8, 1, 64, 1000
    g = torch.Generator("cuda").manual_seed(1)
    q, k, v, do = (torch.randn(T, h * d, device="cuda", generator=g).to(BF16).requires_grad_(True) for h in (hq, hk, hk, hq))
    cu = torch.arange(0, T + 1, S, dtype=torch.int32, device="cuda")
    o = F_.attention(q, k, v, cu, None, S, S, hq, hk, d, True)
    torch.cuda.reset_peak_memory_stats()
    held = torch.cuda.memory_allocated()
    grads = torch.autograd.grad(o, (q, k, v), do, retain_graph=True)
    scratch = torch.cuda.max_memory_allocated() - held - 2 * sum(t.numel() for t in grads)
    assert scratch <= 4 * T * hq + 2 ** 20
    _same(grads, _reference(lambda: torch.autograd.grad(o, (q, k, v), do)))


@pytest.mark.parametrize("scale", [1e-21, 1e-25])
def test_softmax_scales_next_to_nothing(scale):
    """Probabilities that are all but even, and scores that cannot be divided by their scale: P = 1 / keys, dq = dk = 0 but for
    scale times finite sums."""
    from pisceslx_b200.ops import functional as F_
    S, h, d = 300, 2, 64
    g = torch.Generator("cuda").manual_seed(2)
    q, k, v, do = (torch.randn(S, h * d, device="cuda", generator=g).to(BF16).requires_grad_(True) for _ in range(4))
    cu = torch.tensor([0, S], dtype=torch.int32, device="cuda")
    o = F_.attention(q, k, v, cu, None, S, S, h, h, d, False, scale)
    dq, dk, dv = torch.autograd.grad(o, (q, k, v), do)
    rel = lambda a, b: float((a.double() - b).norm() / b.norm())
    # P is rounded to bf16 (2^-9), outputs and gradients once more
    assert rel(o, v.double().mean(0).expand(S, -1)) < 2.0 ** -7 and rel(dv, do.double().mean(0).expand(S, -1)) < 2.0 ** -7
    assert float(dq.abs().max()) <= scale * 1e3 and float(dk.abs().max()) <= scale * 1e3
