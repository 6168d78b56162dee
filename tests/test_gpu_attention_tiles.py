"""Flash attention at the edges of its tiles: items of two 128-query tiles, key blocks of 128, several items per CTA, and the
rotation by 16-byte vectors.  Tolerances: P and dS are rounded to bf16 (2^-9 of each weight), outputs and gradients once more."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30)).item()


def _case(lq, lk, hq, hk, d, causal, seed=0):
    from pisceslx_b200.ops import functional as F_, reference as ref
    g = torch.Generator(device=DEV).manual_seed(seed)
    rand = lambda n, h: torch.randn(n, h * d, device=DEV, generator=g).bfloat16().requires_grad_(True)
    q, k, v = rand(sum(lq), hq), rand(sum(lk), hk), rand(sum(lk), hk)
    cu = lambda lens: torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    do = torch.randn(sum(lq), hq * d, device=DEV, generator=g).bfloat16()
    o = F_.attention(q, k, v, cu(lq), cu(lk), max(lq), max(lk), hq, hk, d, causal)
    got = (o,) + torch.autograd.grad(o, (q, k, v), do)
    f = [t.detach().double().requires_grad_(True) for t in (q, k, v)]
    r = ref.attention_varlen(f[0].view(-1, hq, d), f[1].view(-1, hk, d), f[2].view(-1, hk, d), cu(lq).cpu(), cu(lk).cpu(),
                             causal, 1 / math.sqrt(d)).reshape(-1, hq * d)
    return got, (r,) + torch.autograd.grad(r, f, do.double())


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("lens", [[1, 127, 128, 129], [255, 256, 257, 3], [383, 640, 1]])
@pytest.mark.parametrize("causal", [True, False])
def test_lengths_at_tile_edges(lens, d, causal):
    got, want = _case(lens, lens, 4, 2, d, causal)
    for a, b in zip(got, want):
        assert _rel(a, b) < 6e-3


@pytest.mark.parametrize("lq,lk,causal", [([5, 300], [200, 64], False), ([129, 64], [700, 257], True), ([256], [1], False)])
def test_keys_and_queries_of_unequal_length(lq, lk, causal):
    got, want = _case(lq, lk, 4, 4, 64, causal)
    for a, b in zip(got, want):
        if b.abs().max() < 1e-12:
            # one key: dP equals delta but for the order of 64 products in fp32 (64 x 2^-23 of values up to 16), and up to 256
            # rows of up to 4, scaled by 1/8, add that up
            assert a.isfinite().all() and a.abs().max() < 2e-2
        else:
            assert _rel(a, b) < 6e-3


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("lq,lk,hq,causal", [([1], [129], 2, True), ([64, 128], [257, 384], 4, False), ([1], [2048], 4, True),
                                             ([127], [1000], 8, True), ([512], [512], 4, True), ([385], [640], 4, False),
                                             ([300, 129, 513], [300, 129, 513], 64, True), ([40, 260], [1, 900], 64, True)])
def test_a_lone_query_tile_is_shared_by_both_halves(lq, lk, hq, causal, d):
    """Key tiles dealt out in turn, odd numbers of them among them: with a tile per item and with two."""
    got, want = _case(lq, lk, hq, hq // 2, d, causal, seed=hq)
    for a, b in zip(got, want):
        assert _rel(a, b) < 6e-3


def test_halves_of_very_different_size():
    """One half sees the keys that matter, the other none that does; and halves that are masked entirely."""
    from pisceslx_b200.ops import functional as F_
    g = torch.Generator(device=DEV).manual_seed(5)
    for at in (3, 130, 300):
        q, k, v = (torch.randn(n, 64, device=DEV, generator=g).bfloat16() for n in (100, 384, 384))
        k[at] = q[0] * 8
        q[:] = q[0]
        cu = lambda n: torch.tensor([0, n], dtype=torch.int32, device=DEV)
        o = F_.attention(q, k, v, cu(100), cu(384), 100, 384, 1, 1, 64, False)
        s = q.double() @ k.double().t() / 8
        assert _rel(o, torch.softmax(s, -1) @ v.double()) < 6e-3
        # 100 queries of 40 keys, bottom-right aligned: the first 60 see none
        o = F_.attention(q, k[:40].contiguous(), v[:40].contiguous(), cu(100), cu(40), 100, 40, 1, 1, 64, True)
        assert not o[:60].any() and o.isfinite().all()


def test_several_items_per_cta_with_empty_ones():
    """More items than CTAs; most sequences are far shorter than the longest, so that a CTA passes over items."""
    lens = [1500] + [40 + 13 * i for i in range(24)]
    got, want = _case(lens, lens, 16, 4, 64, True)
    for a, b in zip(got, want):
        assert _rel(a, b) < 6e-3


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_bad_key_reaches_every_query_that_sees_it(bad):
    """Whichever unit computes its exponential, a score that is not finite makes the rows that contain it not finite, and
    no others."""
    from pisceslx_b200.ops import functional as F_
    S, hq, d = 256, 2, 64
    for key in (64, 65, 70, 77, 96):
        q = torch.rand(S, hq * d, device=DEV).bfloat16() + 0.1
        k, v = torch.randn(2, S, hq * d, device=DEV).bfloat16()
        k[key] = bad
        k, v = k.contiguous().requires_grad_(True), v.contiguous().requires_grad_(True)
        q.requires_grad_(True)
        cu = torch.tensor([0, S], dtype=torch.int32, device=DEV)
        o = F_.attention(q, k, v, cu, cu, S, S, hq, hq, d, True)
        dq, dk, dv = torch.autograd.grad(o, (q, k, v), torch.ones_like(o))
        assert o[:key].isfinite().all() and not o[key:].isfinite().any(dim=1).any()
        assert not dq[key:].isfinite().any() and not dv[:key + 1].isfinite().any()


@pytest.mark.parametrize("rot,d,offset", [(64, 64, 0), (128, 128, 0), (32, 64, 0), (64, 64, 2), (24, 64, 0), (16, 16, 0)])
@pytest.mark.parametrize("inverse", [False, True])
def test_rotation_by_vectors_equals_the_reference(rot, d, offset, inverse):
    """Whole vectors, a partial rotation, rows that start off a 16-byte boundary and a width that is no multiple of 16."""
    from pisceslx_b200.ops import kernels, reference as ref
    T, hq, hk = 77, 5, 3
    cos, sin = ref.rope_tables(200, rot, 1e4, device=DEV)
    pos = torch.randint(0, 200, (T,), dtype=torch.int32, device=DEV)
    buf = torch.randn(T, (hq + hk) * d + 8 + offset, device=DEV).bfloat16()
    q, k = buf[:, offset:offset + hq * d], buf[:, offset + hq * d:offset + (hq + hk) * d]
    s = -sin if inverse else sin
    wq = ref.apply_rope(q.reshape(T, hq, d), cos, s, pos, rot).reshape(T, -1)
    wk = ref.apply_rope(k.reshape(T, hk, d), cos, s, pos, rot).reshape(T, -1)
    rest = buf[:, offset + (hq + hk) * d:].clone()
    kernels().rope(q, k, cos, sin, pos, hq, hk, d, rot, inverse)
    # one rounding to bf16 of the same fp32 expression, contracted differently at most
    assert (q.float() - wq.float()).abs().max() <= 2 ** -7 * wq.float().abs().max()
    assert _rel(q, wq) < 1e-3 and _rel(k, wk) < 1e-3
    assert torch.equal(buf[:, offset + (hq + hk) * d:], rest)
