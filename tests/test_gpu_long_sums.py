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


@pytest.mark.parametrize("rows,cols", [(593, 264), (1500, 2056), (1300, 4096), (700, 8192), (1, 64)])
@pytest.mark.parametrize("residual", [False, True])
def test_norm_backward_over_several_rows_a_block(rows, cols, residual):
    """Rows whose loads go out while the row before is summed, and wide ones whose do not; with and without the gradient that
    arrives at the stream."""
    g = torch.Generator("cuda").manual_seed(rows)
    x, dy, res = (torch.randn(rows, cols, device="cuda", generator=g).bfloat16() for _ in range(3))
    w = torch.randn(cols, device="cuda", generator=g).bfloat16()
    rstd = torch.rsqrt(x.float().pow(2).mean(-1) + 1e-6)
    part, dw = torch.empty(min(rows, 592), cols, device="cuda"), torch.empty(cols, device="cuda")
    dx = torch.empty_like(x)
    kernels().rmsnorm_bwd(dy, x, w, rstd, res if residual else None, dx, part, dw, False)
    xhat, gr = x.double() * rstd.double()[:, None], dy.double() * w.double()
    want = rstd.double()[:, None] * (gr - xhat * (gr * xhat).mean(-1, keepdim=True)) + (res.double() if residual else 0.0)
    # one rounding to bf16; sums of `rows` fp32 products
    assert _distance(dx, want) < 2.0 ** -8
    assert _distance(dw, (dy.double() * xhat).sum(0)) < 2.0 ** -20 * max(rows, 8)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("splits", [2, 9, 17, 32])
def test_merge_of_many_key_ranges(splits, d):
    from pisceslx_b200.ops import functional as F_
    g = torch.Generator("cuda").manual_seed(splits)
    B, hq, hk, width = 3, 8, 2, 40
    k, v = (torch.randn(B * width, 64, hk, d, device="cuda", generator=g).bfloat16() for _ in range(2))
    q = torch.randn(B, hq, d, device="cuda", generator=g).bfloat16()
    table = torch.randperm(B * width, device="cuda").int().view(B, width)
    lens = torch.tensor([width * 64, 1, 1111], dtype=torch.int32, device="cuda")
    got = F_.paged_decode(q, k, v, table, lens, splits=splits)
    for b in range(B):
        n = int(lens[b])
        kb, vb = (t[table[b].long()].reshape(-1, hk, d)[:n].double().repeat_interleave(hq // hk, 1) for t in (k, v))
        p = torch.softmax(torch.einsum("hd,nhd->hn", q[b].double(), kb) * d ** -0.5, -1)
        # P and the output are rounded to bf16
        assert _distance(got[b], torch.einsum("hn,nhd->hd", p, vb)) < 6e-3


@pytest.mark.parametrize("rows", [1, 64, 148, 149, 500])
def test_chained_kernels_give_the_bits_of_kernels_run_one_by_one(rows):
    """Norm, product, rotation, cache write, expert layer: with the next kernel starting while the one before ends, with a
    synchronisation after each, and replayed from a graph."""
    from pisceslx_b200.ops import functional as F_, moe as moe_ops, reference as ref
    g = torch.Generator("cuda").manual_seed(rows)
    H, d, E = 256, 64, 8
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, norm, wqkv, wo, gate = rand(rows, H), rand(H), rand(8 * d, H) / 16, rand(H, 4 * d) / 16, rand(E, H)
    w13, w2 = rand(E, 256, H) / 16, rand(E, H, 128) / 11
    cos, sin = ref.rope_tables(rows, d, 1e4, device="cuda")
    pos = torch.arange(rows, dtype=torch.int32, device="cuda")
    pages = torch.zeros(2, (rows + 63) // 64, 64, 2, d, device="cuda", dtype=torch.bfloat16)

    def run(after):
        h, out = x, []
        for _ in range(4):
            n, _none = F_.rms_norm(h, norm)
            after()
            qkv = F_.linear(n, wqkv)
            after()
            q, k, v = qkv[:, :4 * d], qkv[:, 4 * d:6 * d], qkv[:, 6 * d:]
            kernels().rope(q, k, cos, sin, pos, 4, 2, d, d, False)
            after()
            F_.kv_cache_write(k, v, pages[0], pages[1], pos)
            after()
            h = F_.linear(q.contiguous(), wo)
            after()
            weights, idx, counts, _p = moe_ops.gate_topk(F_.linear(h, gate, out_fp32=True), None, 2)
            after()
            h = moe_ops.moe_experts(h, w13, w2, weights, idx, counts, add=n)
            after()
            out += [h, pages.clone()]
        return out

    with torch.no_grad():
        want = run(torch.cuda.synchronize)
        got = run(lambda: None)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            replayed = run(lambda: None)
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    assert all(torch.equal(a, b) for a, b in zip(want, replayed))


@pytest.mark.parametrize("n", [1, 8, 4099, 4104])
@pytest.mark.parametrize("factor", [1.0, 0.25, -3.0])
def test_scaling_of_gradients(n, factor):
    x = torch.randn(n, device="cuda").bfloat16()
    want = (x.float() * factor).bfloat16()
    kernels().scale_(x, torch.tensor([factor], device="cuda"), 1.0)
    assert torch.equal(x, want)
