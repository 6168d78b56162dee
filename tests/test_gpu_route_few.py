"""The router and dispatch plan of few tokens, and the rotation that fills the cache, against the kernels that they take the place
of: the same bits, over edges of the sizes that the rules take."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _gen(seed):
    return torch.Generator("cuda").manual_seed(seed)


@pytest.mark.parametrize("T,E,k", [(1, 1, 1), (1, 64, 6), (2, 8, 2), (15, 33, 5), (16, 64, 6), (16, 256, 8), (16, 200, 16)])
@pytest.mark.parametrize("mode", [(True, 0), (False, 1)])
def test_route_few_equals_gate_and_plan(T, E, k, mode):
    from pisceslx_b200.ops import kernels, moe as M_
    g = _gen(T + E)
    logits, bias = torch.randn(T, E, device="cuda", generator=g), torch.randn(E, device="cuda", generator=g)
    if T == 15:
        logits[:, 7] += 20                                  # one expert that every token takes
    with torch.no_grad():
        w, idx, counts, plan, zero = M_.route_few(logits, bias, k, *mode)
        w0, idx0, counts0, _ = M_.gate_topk(logits, bias, k, *mode)
        rows = M_.padded_rows_bound(T * k, E)
        seg0, tiles0, n0, cur = (torch.empty(n, dtype=torch.int32, device="cuda") for n in (E + 1, rows // 128, 1, E))
        kernels().moe_plan(counts0, seg0, tiles0, n0, cur)
    assert torch.equal(w, w0) and torch.equal(idx, idx0) and torch.equal(counts, counts0) and zero.item() == 0.0 and zero.dim() == 0
    seg, tiles, n, row_map = plan.split([E + 1, rows // 128, 1, T * k])
    assert torch.equal(seg, seg0) and torch.equal(n, n0) and torch.equal(tiles[:int(n)], tiles0[:int(n)])
    # every expert's assignments fill its segment from the front, each row once
    want = torch.cat([torch.arange(int(s), int(s) + int(c)) for s, c in zip(seg0[:E].tolist(), counts0.tolist())])
    assert torch.equal(row_map.cpu().long().sort().values, want)
    assert (seg[idx.long().flatten()] <= row_map).all() and (row_map < seg[idx.long().flatten() + 1]).all()


def test_more_tokens_go_to_the_general_kernels():
    from pisceslx_b200.ops import moe as M_
    with torch.no_grad():
        assert M_.route_few(torch.randn(17, 8, device="cuda"), None, 2) is None
    assert M_.route_few(torch.randn(4, 8, device="cuda"), None, 2) is None            # with a gradient


def test_route_few_of_nan_and_infinities():
    from pisceslx_b200.ops import moe as M_
    logits = torch.randn(4, 8, device="cuda", generator=_gen(0))
    logits[1] = float("nan")
    logits[2] = float("-inf")
    logits[3, 2:] = float("-inf")
    with torch.no_grad():
        w, idx, counts, _, _ = M_.route_few(logits, None, 3)
    assert ((idx >= 0) & (idx < 8)).all() and int(counts.sum()) == 12
    assert w[1].isnan().all() and w[0].isfinite().all() and idx[3, 0] < 2 and idx[3, 1] < 2


def test_experts_with_a_plan_and_without():
    from pisceslx_b200.ops import moe as M_
    g = _gen(5)
    x = torch.randn(16, 256, device="cuda", generator=g).to(BF16)
    w13 = (torch.randn(16, 256, 256, device="cuda", generator=g) / 16).to(BF16)
    w2 = (torch.randn(16, 256, 128, device="cuda", generator=g) / 12).to(BF16)
    with torch.no_grad():
        w, idx, counts, plan, _ = M_.route_few(torch.randn(16, 16, device="cuda", generator=g), None, 4)
        for few in (True, False):
            assert torch.equal(M_.moe_experts(x, w13, w2, w, idx, counts, few=few, plan=plan),
                               M_.moe_experts(x, w13, w2, w, idx, counts, few=few))


@pytest.mark.parametrize("T,hq,hk,d,rot,pad", [(1, 32, 8, 128, 128, 0), (65, 4, 2, 64, 64, 0), (300, 8, 1, 128, 128, 8), (5, 4, 4, 80, 80, 0),
                                               (7, 4, 2, 128, 64, 0), (9, 2, 2, 32, 32, 0)])
def test_rope_cache_equals_rotation_and_write(T, hq, hk, d, rot, pad):
    """Whole heads by vectors; partial rotations and narrow heads by the two kernels.  Tokens without a slot are not written; a
    slot past the end is reported and skipped."""
    from pisceslx_b200.ops import functional as F_, check_status, kernels, status_word
    from pisceslx_b200.ops.reference import rope_tables
    g = _gen(T)
    cos, sin = rope_tables(512, rot, 1e4, device="cuda")
    pos = torch.randint(0, 512, (T,), device="cuda", generator=g, dtype=torch.int32)
    slots = torch.randperm(512, device="cuda", generator=g)[:T].int()
    slots[::3] = torch.where(torch.arange(T, device="cuda")[::3] % 2 == 0, -1, slots[::3])
    if T > 60:
        slots[1] = 512
    buf = torch.randn(T, (hq + 2 * hk) * d + pad, device="cuda", generator=g).to(BF16)
    out = []
    for fused in (True, False):
        x = buf.clone()
        q, k, v = x[:, :hq * d], x[:, hq * d:(hq + hk) * d], x[:, (hq + hk) * d:(hq + 2 * hk) * d]
        kc, vc = (torch.zeros(8, 64, hk, d, device="cuda", dtype=BF16) for _ in range(2))
        if fused:
            F_.rope_cache(q, k, v, cos, sin, pos, hq, hk, d, rot, kc, vc, slots)
        else:
            kernels().rope(q, k, cos, sin, pos, hq, hk, d, rot, False)
            F_.kv_cache_write(k, v, kc, vc, slots)
        word = int(status_word(x.device)[0])
        assert word == (8 if T > 60 else 0)
        status_word(x.device).zero_()
        out.append((x, kc, vc))
    assert all(torch.equal(a, b) for a, b in zip(*out))


def test_cache_rows_off_16_bytes_are_refused():
    from pisceslx_b200.ops import functional as F_
    k = torch.zeros(3, 132, device="cuda", dtype=BF16)[:, :128]
    cache = torch.zeros(2, 64, 2, 64, device="cuda", dtype=BF16)
    with pytest.raises(RuntimeError):
        F_.kv_cache_write(k, k, cache, cache.clone(), torch.zeros(3, device="cuda", dtype=torch.int32))


@pytest.mark.parametrize("hq,hk,d,page,extra", [(32, 8, 128, 64, 64), (4, 4, 64, 64, 8), (8, 2, 64, 64, 4), (6, 2, 64, 64, 8), (8, 1, 128, 16, 8)])
def test_decode_reads_queries_inside_a_projection(hq, hk, d, page, extra):
    """A row pitch of whole and of broken vectors, a group and a page that the tensor-core kernel does not take."""
    from pisceslx_b200.ops import functional as F_
    g = _gen(hq)
    B = 3
    buf = torch.randn(B, hq * d + extra, device="cuda", generator=g).to(BF16)
    kc, vc = (torch.randn(12, page, hk, d, device="cuda", generator=g).to(BF16) for _ in range(2))
    table = torch.arange(12, device="cuda", dtype=torch.int32).view(3, 4)
    lens = torch.tensor([1, page + 3, 4 * page], device="cuda", dtype=torch.int32)
    q = buf[:, :hq * d].view(B, hq, d)
    if (hq // hk) & (hq // hk - 1):
        with pytest.raises(RuntimeError):
            F_.paged_decode(q, kc, vc, table, lens)
        return
    assert torch.equal(F_.paged_decode(q, kc, vc, table, lens), F_.paged_decode(q.contiguous(), kc, vc, table, lens))


def test_a_plan_is_for_the_numbers_that_the_router_returned():
    """A router whose numbers are exchanged, or written to, after it has planned: the layer plans for itself."""
    from pisceslx_b200 import YvConfig
    from pisceslx_b200.models.moe_layer import YvDeepSeekMoELayer
    torch.manual_seed(0)
    cfg = YvConfig.tiny_text_moe()
    layer = YvDeepSeekMoELayer(cfg, 0).to("cuda", BF16).eval()
    x = torch.randn(9, cfg.hidden_size, device="cuda").to(BF16)
    route = layer.router.forward
    with torch.inference_mode():
        served = layer(x)[0].clone()
    with torch.no_grad():
        plain = layer(x)[0]
        assert layer.router.last_plan is not None and torch.equal(served, plain)

        def exchanged(y):
            w, idx, aux = route(y)
            return w.flip(1), idx.flip(1), aux

        def written(y):
            w, idx, aux = route(y)
            idx.copy_(idx.flip(1))
            return w.flip(1), idx, aux

        for forward in (exchanged, written):
            layer.router.forward = forward
            got = layer(x)[0]                              # the same sums in another order
            assert float((got.float() - plain.float()).norm() / plain.float().norm()) < 1e-2


@pytest.mark.parametrize("mode", [torch.no_grad, torch.inference_mode])
@pytest.mark.parametrize("tokens", [1, 9, 16])
def test_no_plan_outlives_a_write_to_its_numbers(mode, tokens):
    """Numbers written to in place between the router and the experts, where tensors have versions and where they have none."""
    from pisceslx_b200 import YvConfig
    from pisceslx_b200.models.moe_layer import YvDeepSeekMoELayer
    torch.manual_seed(0)
    cfg = YvConfig.tiny_text_moe()
    layer = YvDeepSeekMoELayer(cfg, 0).to("cuda", BF16).eval()
    x = torch.randn(tokens, cfg.hidden_size, device="cuda").to(BF16)
    route = layer.router.forward

    def written(y):
        w, idx, aux = route(y)
        idx.copy_(idx.flip(1))
        return w.flip(1), idx, aux

    with mode():
        plain = layer(x)[0]
        layer.router.forward = written
        got = layer(x)[0]                                  # the same sums in another order
    assert float((got.float() - plain.float()).norm() / plain.float().norm()) < 1e-2


@pytest.mark.parametrize("low", [float("-inf"), float("nan"), torch.finfo(torch.float32).min])
@pytest.mark.parametrize("E,k,alone", [(8, 3, [[1, 2], [2, 1], [7], [0], [3, 4, 5], []]), (70, 16, [[69, 33, 1, 0], [32], [2, 1], []]), (2, 2, [[1], []])])
@pytest.mark.parametrize("few", [True, False])
def test_no_expert_is_taken_twice(low, E, k, alone, few):
    """Fewer experts with a logit than are taken: the others come lowest first, without a weight."""
    from pisceslx_b200.ops import moe as M_
    logits = torch.full((len(alone), E), low)
    for t, experts in enumerate(alone):
        for j, e in enumerate(experts):
            logits[t, e] = 2.0 - j
    with torch.no_grad():
        w, idx, counts = (M_.route_few if few else M_.gate_topk)(logits.cuda(), None, k)[:3]
    want = [experts[:k] + [e for e in range(E) if e not in experts][:max(k - len(experts), 0)] for experts in alone]
    assert idx.tolist() == want and counts.tolist() == torch.bincount(torch.tensor(want).flatten(), minlength=E).tolist()
    for t, experts in enumerate(alone):
        if experts and low == low:                          # NaN leaves no weights
            shares = torch.softmax(torch.tensor([2.0 - j for j in range(len(experts))]), 0)
            torch.testing.assert_close(w[t].cpu()[:len(experts)], shares / shares.sum(), rtol=1e-5, atol=0)
            assert not w[t, len(experts):].any()


@pytest.mark.parametrize("pitch", [132, 129])
def test_a_single_cache_row_has_no_pitch(pitch):
    """One token's row out of a buffer whose rows are no whole number of 16-byte pieces, with a rotation and without."""
    from pisceslx_b200.ops import functional as F_
    from pisceslx_b200.ops.reference import rope_tables
    k, v = (torch.randn(1, pitch, device="cuda", generator=_gen(i)).to(BF16)[:, :128] for i in range(2))
    assert k.stride(0) == pitch
    slot, pos = torch.tensor([70], device="cuda", dtype=torch.int32), torch.tensor([0], device="cuda", dtype=torch.int32)
    cos, sin = rope_tables(8, 64, 1e4, device="cuda")
    for rotate in (False, True):
        kc, vc = (torch.zeros(2, 64, 2, 64, device="cuda", dtype=BF16) for _ in range(2))
        if rotate:                                          # by nothing at place 0
            F_.rope_cache(k.clone(), k, v, cos, sin, pos, 2, 2, 64, 64, kc, vc, slot)
        else:
            F_.kv_cache_write(k, v, kc, vc, slot)
        for cache, row in ((kc, k), (vc, v)):
            assert torch.equal(cache[1, 6].flatten(), row[0]) and int((cache != 0).sum()) == int((row != 0).sum())


def test_a_slot_map_longer_than_the_tokens():
    """Slots of a whole bucket with fewer tokens: the first of them count, as for kv_cache_write; fewer slots than tokens are refused."""
    from pisceslx_b200.ops import functional as F_
    from pisceslx_b200.ops.reference import rope_tables
    q, k, v = (torch.randn(3, 256, device="cuda", generator=_gen(i)).to(BF16) for i in range(3))
    cos, sin = rope_tables(8, 128, 1e4, device="cuda")
    pos, slots = torch.arange(3, device="cuda", dtype=torch.int32), torch.tensor([5, 70, 6, 90, -1], device="cuda", dtype=torch.int32)
    out = []
    for n in (3, 5):
        kc, vc = (torch.zeros(2, 64, 2, 128, device="cuda", dtype=BF16) for _ in range(2))
        F_.rope_cache(q.clone(), k.clone(), v, cos, sin, pos, 2, 2, 128, 128, kc, vc, slots[:n])
        out.append((kc, vc))
    assert all(torch.equal(a, b) for a, b in zip(*out))
    with pytest.raises(RuntimeError):
        F_.rope_cache(q.clone(), k.clone(), v, cos, sin, pos, 2, 2, 128, 128, *out[0], slots[:2])
