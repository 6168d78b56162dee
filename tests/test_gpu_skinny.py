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
                                          (200, 16, 520, 128, True)])
def test_experts_without_gradient_match_fp64(T, E, H, F, same):
    """Few tokens, odd widths, and all tokens at the same experts: more than one pass and more than one tile each."""
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
