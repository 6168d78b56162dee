"""Long sums over few outputs: the loss's gradient split along the vocabulary, column sums, the scaling of gradients."""
import pytest
import torch

from pisceslx_b200.ops import kernels, loss, status_word

pytestmark = pytest.mark.gpu


def _distance(a: torch.Tensor, b: torch.Tensor) -> float:
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("M,N,K", [(1, 64, 4096), (129, 136, 4104), (128, 256, 8200), (300, 1024, 20000)])
def test_split_product_matches_fp64(M, N, K):
    """Row and column remainders, and a last slice that ends inside a step of 64."""
    assert loss._slices(M, N, K) > 1
    g = torch.Generator("cuda").manual_seed(M)
    dl = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = torch.randn(K, N, device="cuda", generator=g).bfloat16()
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    loss._times_weights(dl, w, out, status_word(dl.device))
    # one rounding to bf16; fp32 sums stay far below it
    assert _distance(out, dl.double() @ w.double()) < 2.0 ** -8


def test_split_line():
    assert loss._slices(8192, 4096, 32000) == 1 and loss._slices(256, 256, 1024) == 1 and loss._slices(64, 66, 1 << 16) == 1


@pytest.mark.parametrize("rows,cols", [(1, 8), (17, 264), (700, 40)])
def test_norm_weight_gradient_matches_fp64(rows, cols):
    g = torch.Generator("cuda").manual_seed(rows)
    x, dy = (torch.randn(rows, cols, device="cuda", generator=g).bfloat16() for _ in range(2))
    w = torch.ones(cols, device="cuda").bfloat16()
    rstd = torch.rsqrt(x.float().pow(2).mean(-1) + 1e-6)
    part = torch.empty(min(rows, 592), cols, device="cuda")
    dw = torch.empty(cols, device="cuda")
    kernels().rmsnorm_bwd(dy, x, w, rstd, None, torch.empty_like(x), part, dw, False)
    want = (dy.double() * x.double() * rstd.double()[:, None]).sum(0)
    # sums of `rows` fp32 products
    assert _distance(dw, want) < 2.0 ** -20 * max(rows, 8)


@pytest.mark.parametrize("n", [1, 8, 4099, 4104])
@pytest.mark.parametrize("factor", [1.0, 0.25, -3.0])
def test_scaling_of_gradients(n, factor):
    x = torch.randn(n, device="cuda").bfloat16()
    want = (x.float() * factor).bfloat16()
    kernels().scale_(x, torch.tensor([factor], device="cuda"), 1.0)
    assert torch.equal(x, want)
