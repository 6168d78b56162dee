"""The differentiable operators of a decoder layer (csrc/binding_autograd.inc) against plain fp32 math: shapes and strides that the
kernels do not take as they come, parts of the gradients, saved-tensor hooks, and transforms that stay refused."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


def _ops():
    from pisceslx_b200.ops import functional as F_, moe as M_, reference as ref
    return F_, M_, ref


def _gen(seed):
    g = torch.Generator("cuda").manual_seed(seed)
    return lambda *s: torch.randn(*s, device="cuda", generator=g)


# the layouts in which an activation [2, 5, 256] may come: as it is, a column range of a wider buffer, every other row, transposed
LAYOUTS = {"plain": lambda r: r(2, 5, 256), "columns": lambda r: r(2, 5, 512)[..., 64:320], "rows": lambda r: r(2, 10, 256)[:, ::2],
           "transposed": lambda r: r(5, 2, 256).transpose(0, 1), "inner": lambda r: r(2, 256, 5).transpose(1, 2)}


@pytest.mark.parametrize("layout", LAYOUTS)
def test_linear_norm_and_activation_over_layouts(layout):
    F_, _, ref = _ops()
    r = _gen(1)
    x0 = LAYOUTS[layout](r).to(BF16)
    w0, n0, mix0 = (r(384, 256) / 16).to(BF16), (1 + 0.1 * r(256)).to(BF16), r(2).abs()

    def run(dtype, linear, norm, mix):
        x = x0.detach().to(dtype).requires_grad_(True) if dtype != BF16 else x0.detach().requires_grad_(True)
        w, n, m = (t.detach().to(dtype).requires_grad_(True) for t in (w0, n0, mix0))
        m = mix0.detach().clone().requires_grad_(True)
        y, s = norm(x, n, x)
        z = mix(linear(y, w).reshape(-1, 384), m)
        out = (z.float().sin().sum() + s.float().cos().sum())
        return z, torch.autograd.grad(out, (x, w, n, m))

    got = run(BF16, F_.linear, lambda x, n, res: F_.rms_norm(x, n, 1e-6, res), F_.swiglu_mix)

    def mix32(y, m):
        g, u = y.chunk(2, -1)
        return (torch.nn.functional.silu(g) * u).view(-1, 2, 192).mul(m.view(1, 2, 1)).view(-1, 192)
    want = run(torch.float32, torch.nn.functional.linear,
               lambda x, n, res: (ref.rms_norm(x + res, n, 1e-6), x + res), mix32)
    assert rel(got[0], want[0]) < 2e-2                     # three roundings to bf16 on the way
    for a, b in zip(got[1], want[1]):
        assert a.shape == b.shape and rel(a, b) < 3e-2


@pytest.mark.parametrize("needs", [(True, False), (False, True)])
def test_only_the_gradients_asked_for(needs):
    F_, _, _ = _ops()
    r = _gen(2)
    x, w = r(130, 256).to(BF16).requires_grad_(needs[0]), r(64, 256).to(BF16).requires_grad_(needs[1])
    F_.linear(x, w).sum().backward()
    assert (x.grad is not None) == needs[0] and (w.grad is not None) == needs[1]


@pytest.mark.parametrize("T,E,k,deterministic", [(1, 4, 2, False), (129, 4, 2, True), (300, 8, 3, False)])
def test_router_and_experts_match_the_oracle(T, E, k, deterministic):
    _, M_, ref = _ops()
    r = _gen(T)
    x, w13, w2 = (t.to(BF16).requires_grad_(True) for t in (r(T, 128), r(E, 256, 128) / 11, r(E, 128, 128) / 11))
    add, logits = r(T, 128).to(BF16).requires_grad_(True), r(T, E).requires_grad_(True)
    w, idx, counts, probs = M_.gate_topk(logits, None, k)
    assert not (idx.requires_grad or counts.requires_grad or probs.requires_grad)
    out = M_.moe_experts(x, w13, w2, w, idx, counts, deterministic, add=add)
    f = [t.detach().float().requires_grad_(True) for t in (x, w13, w2, add, logits)]
    wr, ir, _, _ = ref.gate_topk(f[4], None, k)
    assert torch.equal(ir.int(), idx)
    want = ref.moe_experts(f[0], f[1], f[2], wr, idx.long()) + f[3]
    assert rel(out, want) < 1.5e-2
    do = r(T, 128)
    got_g = torch.autograd.grad(out, (x, w13, w2, add, logits), do.to(BF16))
    for a, b in zip(got_g, torch.autograd.grad(want, f, do.to(BF16).float())):
        assert rel(a, b) < 2.5e-2


def test_saved_tensors_pass_the_hooks_and_transforms_stay_refused():
    F_, _, _ = _ops()
    r = _gen(3)
    x, w = r(40, 256).to(BF16).requires_grad_(True), r(64, 256).to(BF16).requires_grad_(True)
    seen = []

    def pack(t):
        seen.append(tuple(t.shape))
        return t.cpu()

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        y = F_.linear(x, w)
    a = torch.autograd.grad(y, (x, w), torch.ones_like(y))
    assert seen == [(40, 256), (64, 256)]
    y = F_.linear(x, w)
    assert all(torch.equal(p, q) for p, q in zip(a, torch.autograd.grad(y, (x, w), torch.ones_like(y))))
    with pytest.raises(RuntimeError):                      # a saved operand that was written to
        y = F_.linear(x, w)
        w.data.add_(0)
        with torch.no_grad():
            w.add_(1)
        y.sum().backward()
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: F_.linear(t, w.detach()).sum())(x.detach())
    import torch.autograd.forward_ad as fw
    with pytest.raises((RuntimeError, NotImplementedError)), fw.dual_level():
        F_.linear(fw.make_dual(x.detach(), torch.ones_like(x)), w.detach())


@pytest.mark.parametrize("T,V,H", [(1, 5, 8), (32, 4000, 264), (33, 1, 2056), (95, 2, 128), (2049, 7, 64), (4100, 100000, 40)])
def test_embedding_gradient(T, V, H):
    """Runs of equal words within a block of 32 places, over its edges and over many blocks; chunks of 2048 comparisons."""
    F_, _, _ = _ops()
    r = _gen(T)
    w = r(V, H).to(BF16).requires_grad_(True)
    ids = torch.randint(0, V, (1, T), device="cuda", generator=torch.Generator("cuda").manual_seed(V))
    y = F_.embedding(ids, w)
    assert torch.equal(y, torch.nn.functional.embedding(ids, w))
    dy = r(1, T, H).to(BF16)
    grads = [torch.autograd.grad(F_.embedding(i, w), w, dy)[0] for i in (ids, ids, ids.int())]
    assert all(torch.equal(grads[0], g) for g in grads[1:])
    want = torch.zeros(V, H, device="cuda", dtype=torch.float64).index_add_(0, ids[0], dy[0].double())
    # one rounding to bf16 of sums whose fp32 additions err far less
    assert ((grads[0].double() - want).abs() <= want.abs() * 2.0 ** -8 + T * 2.0 ** -22).all()
    assert (grads[0][want.abs().sum(1) == 0] == 0).all()


@pytest.mark.parametrize("T,V,H", [(300, 1000, 128), (513, 5000, 256)])
def test_loss_in_one_chunk_and_in_several(T, V, H):
    """The same sums in another order: the weight gradient is rounded to bf16 once either way, the rest row by row."""
    from pisceslx_b200.ops.loss import linear_cross_entropy
    r = _gen(T)
    h, w = r(T, H).to(BF16).requires_grad_(True), (r(V, H) * H ** -0.5).to(BF16).requires_grad_(True)
    labels = torch.randint(0, V, (T,), device="cuda", generator=torch.Generator("cuda").manual_seed(V))
    labels[::7] = -100
    out = []
    for chunk in (128, T):
        loss = linear_cross_entropy(h, w, labels, -100, None, chunk)
        out.append((loss, *torch.autograd.grad(loss, (h, w))))
    for a, b in zip(*out):
        assert rel(a, b) < 2.0 ** -8


@pytest.mark.parametrize("off", [1, 4, 8])
def test_embedding_gradient_off_16_bytes(off):
    """A gradient that is contiguous but begins between 16-byte boundaries (or, at 8, on one)."""
    F_, _, _ = _ops()
    r = _gen(off)
    T, V, H = 70, 50, 64
    w = r(V, H).to(BF16).requires_grad_(True)
    ids = torch.randint(0, V, (T,), device="cuda", generator=torch.Generator("cuda").manual_seed(V))
    dy = r(T * H + off).to(BF16)[off:].view(T, H)
    got, = torch.autograd.grad(F_.embedding(ids, w), w, dy)
    want = torch.zeros(V, H, device="cuda", dtype=torch.float64).index_add_(0, ids, dy.double())
    assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + T * 2.0 ** -22).all()


def test_embedding_under_transforms_and_twice():
    """What torch's embedding does, the model's does too: function transforms, forward mode, a gradient of a gradient."""
    import torch.autograd.forward_ad as fw
    from pisceslx_b200.models.model import YvTokenEmbedding
    r = _gen(3)
    ids = torch.tensor([1, 2, 2, 7], device="cuda")
    layer = YvTokenEmbedding(8, 64, device="cuda", dtype=BF16)
    plain = torch.nn.Embedding(8, 64, device="cuda", dtype=BF16)
    plain.load_state_dict(layer.state_dict())
    tangent, seed = r(8, 64).to(BF16), r(4, 64).to(BF16)

    def results(m):
        w = m.weight
        call = lambda t: torch.func.functional_call(m, {"weight": t}, (ids,))
        with fw.dual_level():
            forward = fw.unpack_dual(call(fw.make_dual(w, tangent))).tangent
        first, = torch.autograd.grad((m(ids).float() ** 3).sum(), w, create_graph=True)
        second, = torch.autograd.grad((first.float() * tangent.float()).sum(), w)
        return [torch.func.grad(lambda t: (call(t).float() * seed.float()).sum())(w), forward, first, second,
                torch.func.vmap(call)(torch.stack([w, 2 * w])), torch.func.jvp(call, (w,), (tangent,))[1]]

    for a, b in zip(results(layer), results(plain)):
        assert torch.equal(a, b)


def test_router_and_experts_refuse_other_ranks():
    """Tokens of several sequences that have not been flattened: sizes taken from the wrong dimensions would reach the kernels."""
    _, M_, _ = _ops()
    r = _gen(4)
    w13, w2, x = r(4, 256, 128).to(BF16), r(4, 128, 128).to(BF16), r(2, 3, 128).to(BF16)
    for logits in (r(2, 3, 4), r(4)):
        for grad in (True, False):
            with torch.set_grad_enabled(grad), pytest.raises((ValueError, IndexError)):
                M_.gate_topk(logits, None, 2)
    w, idx, counts, _ = M_.gate_topk(r(6, 4), None, 2)
    for bad in ((x, w13, w2, w, idx), (x.view(6, 128), w13[None], w2, w, idx), (x.view(6, 128), w13, w2[0], w, idx),
                (x.view(6, 128), w13, w2, w, idx.view(2, 3, 2)), (x, w13, w2, w, idx.view(2, 6))):
        for grad in (True, False):
            with torch.set_grad_enabled(grad), pytest.raises((ValueError, IndexError)):
                M_.moe_experts(*bad, counts)
