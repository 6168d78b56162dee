"""Products of few token rows with large weights against fp64, at the edges of their tiles."""
import pytest
import torch

from pisceslx_b200.ops import functional as F_
from pisceslx_b200.ops import moe as moe_ops

pytestmark = pytest.mark.gpu
# rounding of the result to bf16 is at most 2^-9 of a value; sums of K products in fp32 stay below 2^-20 of the result's norm
LIMIT = {torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -18}


def _distance(a: torch.Tensor, b: torch.Tensor) -> float:
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("N,K", [(8, 64), (100, 520), (128, 8), (129, 2048), (4096, 256), (19000, 128)])
@pytest.mark.parametrize("M", [1, 16, 17, 64, 65, 128])
def test_rows_match_fp64_and_do_not_depend_on_their_neighbours(M, N, K):
    g = torch.Generator("cuda").manual_seed(M * 7 + N)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = torch.randn(N, K, device="cuda", generator=g).bfloat16()
    b = torch.randn(N, device="cuda", generator=g).bfloat16()
    want = x.double() @ w.double().t()
    for dtype in LIMIT:
        y = F_.gemm_skinny(x, w, None, dtype)
        assert y.dtype == dtype and _distance(y, want) < LIMIT[dtype]
        assert torch.equal(F_.gemm_skinny(x[M - 1:], w, None, dtype), y[M - 1:])
    assert _distance(F_.gemm_skinny(x, w, b), want + b.double()) < LIMIT[torch.bfloat16]
    wide = torch.randn(N, K + 8, device="cuda", generator=g).bfloat16()[:, :K]      # a row pitch
    assert _distance(F_.gemm_skinny(x, wide), x.double() @ wide.double().t()) < LIMIT[torch.bfloat16]


@pytest.mark.parametrize("T,E,H,F,same", [(1, 8, 256, 64, False), (17, 8, 264, 192, False), (130, 4, 128, 64, False),
                                          (200, 16, 520, 128, True), (100, 16, 264, 128, True)])
def test_experts_without_gradient_match_fp64(T, E, H, F, same):
    """Few tokens, odd widths, and all tokens at the same experts: 200 fill more than one tile, 100 more than the 64 slots of a
    pass."""
    g = torch.Generator("cuda").manual_seed(T)
    x = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    w13 = (torch.randn(E, 2 * F, H, device="cuda", generator=g) * H ** -0.5).bfloat16()
    w2 = (torch.randn(E, H, F, device="cuda", generator=g) * F ** -0.5).bfloat16()
    idx = torch.rand(T, E, device="cuda", generator=g).topk(2, -1).indices.int()
    if same:
        idx[:] = torch.tensor([3, 5], device="cuda", dtype=torch.int32)
    weights = torch.rand(T, 2, device="cuda", generator=g)
    assert moe_ops._few_tokens(2 * T, w13, w2)
    with torch.no_grad():
        got = moe_ops.moe_experts(x, w13, w2, weights, idx)
    want = torch.zeros(T, H, device="cuda", dtype=torch.float64)
    for t in range(T):
        for j in range(2):
            e = int(idx[t, j])
            gate, up = (w13[e].double() @ x[t].double()).chunk(2)
            want[t] += float(weights[t, j]) * (w2[e].double() @ (torch.nn.functional.silu(gate) * up))
    # the activation, the experts' outputs and their sum are rounded to bf16
    assert _distance(got, want) < 3 * 2.0 ** -8


@pytest.mark.parametrize("M,H,seg,parts", [(1, 64, 64, 1), (17, 520, 64, 3), (128, 256, 192, 2), (130, 256, 64, 2)])
def test_shared_experts_activation_matches_fp64(M, H, seg, parts):
    """silu(gate) * up times a weight per expert: inside the product (up to 128 rows) and by itself, with its gradients."""
    g = torch.Generator("cuda").manual_seed(M)
    x = torch.randn(M, H, device="cuda", generator=g).bfloat16()
    w = (torch.randn(parts * 2 * seg, H, device="cuda", generator=g) * H ** -0.5).bfloat16()
    mix = torch.softmax(torch.randn(parts, device="cuda", generator=g), 0).bfloat16()
    y = (x.double() @ w.double().t()).view(M, parts, 2, seg)
    want = torch.nn.functional.silu(y[:, :, 0]) * y[:, :, 1] * mix.double()[:, None]
    inside = F_.skinny_swiglu(x, w, seg, mix)
    assert (inside is None) == (M > 128)
    if inside is not None:
        assert _distance(inside.view_as(want), want) < 2.0 ** -8
    y16 = F_.linear(x, w).view(M * parts, 2 * seg).detach().requires_grad_(True)
    mix32 = mix.float().requires_grad_(True)
    out = F_.swiglu_mix(y16, mix32)
    grad = torch.randn(out.shape, device="cuda", generator=g).bfloat16()
    got = torch.autograd.grad(out, (y16, mix32), grad)
    y64, mix64 = y16.detach().double().requires_grad_(True), mix32.detach().double().requires_grad_(True)
    a, b = y64.chunk(2, -1)
    out64 = torch.nn.functional.silu(a) * b * mix64.repeat(M)[:, None]
    ref = torch.autograd.grad(out64, (y64, mix64), grad.double())
    assert _distance(out.detach(), out64.detach()) < 2.0 ** -8 and _distance(got[0], ref[0]) < 2.0 ** -8
    # __expf and sums of M x seg products in fp32, of which some cancel
    assert got[1].dtype == torch.float32 and _distance(got[1], ref[1]) < 1e-4


@pytest.mark.parametrize("T", [1, 147, 148])
def test_combine_adds_the_shared_experts(T):
    g = torch.Generator("cuda").manual_seed(T)
    E, H, F, k = 8, 1152, 64, 3
    x = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    w13 = (torch.randn(E, 2 * F, H, device="cuda", generator=g) * H ** -0.5).bfloat16()
    w2 = (torch.randn(E, H, F, device="cuda", generator=g) * F ** -0.5).bfloat16()
    idx = torch.rand(T, E, device="cuda", generator=g).topk(k, -1).indices.int()
    weights = torch.rand(T, k, device="cuda", generator=g)
    add = torch.randn(T, H, device="cuda", generator=g).bfloat16().requires_grad_(True)
    alone = moe_ops.moe_experts(x, w13, w2, weights, idx)
    both = moe_ops.moe_experts(x, w13, w2, weights, idx, add=add)
    # both results are rounded
    assert _distance(both.detach(), alone.double() + add.detach().double()) < 2 * 2.0 ** -8
    grad = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    assert torch.equal(torch.autograd.grad(both, add, grad)[0], grad)


@pytest.mark.parametrize("slots", [1, 16, 32, 64, 128])
def test_passes_over_a_tile(slots):
    """Tiles of 1 to 128 tokens in passes of 16 to 128: each pass reads the weights again, takes the next tokens and the other
    accumulator."""
    from pisceslx_b200.ops import kernels, status_word
    g = torch.Generator("cuda").manual_seed(slots)
    tokens, H, F = [17, 128, 1, 0, 65, 129, 100], 264, 192
    E, T = len(tokens), sum(tokens)
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(tokens))[torch.randperm(T)].cuda().int()[:, None].contiguous()
    x = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    w13 = (torch.randn(E, 2 * F, H, device="cuda", generator=g) * H ** -0.5).bfloat16()
    counts = torch.tensor(tokens, dtype=torch.int32, device="cuda")
    xp, plan = moe_ops.permute_tokens(x, idx, counts, E, False, False)
    layout = (plan.tile_expert, plan.num_m_tiles, plan.seg_offsets, counts, slots)
    y = torch.full((xp.shape[0], 2 * F), float("nan"), device="cuda", dtype=torch.bfloat16)
    act = torch.full((xp.shape[0], F), float("nan"), device="cuda", dtype=torch.bfloat16)
    kernels().gemm_skinny_grouped(xp, w13, y, *layout, False, status_word(x.device))
    kernels().gemm_skinny_grouped(xp, w13, act, *layout, True, status_word(x.device))
    rows = plan.row_map[:, 0].long()
    want = torch.einsum("th,tnh->tn", x.double(), w13[idx[:, 0].long()].double())
    gate, up = want.chunk(2, -1)
    assert _distance(y[rows], want) < 2.0 ** -8
    assert _distance(act[rows], torch.nn.functional.silu(gate) * up) < 2.0 ** -8


@pytest.mark.parametrize("N,K", [(6144, 4096), (4500, 4096), (9216, 3072), (37888, 256), (40000, 128)])
def test_sizes_whose_clusters_fill_the_chip(N, K):
    """One cluster more than fits at six, eight and four slices, the most tiles that fit, and more than fit."""
    g = torch.Generator("cuda").manual_seed(N)
    w = torch.randn(N, K, device="cuda", generator=g).bfloat16()
    for M in (1, 128):
        x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
        y = F_.linear(x, w)
        assert _distance(y, x.double() @ w.double().t()) < LIMIT[torch.bfloat16]
        assert torch.equal(F_.linear(x[M - 1:], w), y[M - 1:])
