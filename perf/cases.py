"""Performance cases of the framework's main path: training and serving of the Yv mixture-of-experts text models.

Six kinds of work, each through the call that a program makes:

* ``train``      forward and backward of a model (``build_model``; the call that a trainer makes per micro-batch);
* ``attention``  forward and backward of ``ops.functional.rope_attention`` over packed sequences: one layer's attention in
                 training, from short documents to a long sequence;
* ``images``     forward and backward of ``ops.functional.attention``, not causal: the vision encoder over image patches;
* ``prefill``    a prompt through ``YvInferenceEngine.run_tokens`` (time to first token);
* ``decode``     one token for every running sequence through the engine's decode runner;
* ``optimizer``  one Muon / AdamW step over given gradients.

Models have the sizes of the repository's presets; depth is cut to a few layers (all layers of a model are alike) and, for
the wide model, the vocabulary to 32000, which keeps the share of the output head near what it is at full depth.  Weights
have the scale at which a trained network works."""
from __future__ import annotations

import math
import random
from typing import Any, Dict, List, Optional

import torch

from pisceslx_b200 import YvConfig
from pisceslx_b200.models import build_model
from pisceslx_b200.models.cache_policies import YvSpeculativeCacheManager
from pisceslx_b200.ops import functional as F_
from pisceslx_b200.ops.reference import rope_tables
from pisceslx_b200.optim import build_optimizer
from pisceslx_b200.optim.muon import NS_COEFFS
from pisceslx_b200.serve.engine import YvEngineConfig, YvInferenceEngine

DEV = "cuda"
BF16 = torch.bfloat16
PAGE = 64                       # tokens per cache page, the engine's default
LR = 0.02


def listed() -> List[Dict[str, Any]]:
    wide = dict(preset="7b", vocab=32000)
    return [
        # the smallest preset at the batch of the repository's CPU benchmark: launches and latency count
        dict(name="train_tiny", kind="train", preset="tiny", layers=4, vocab=154856, batch=2, seq=256),
        # the 0.5B preset (experts of 704), odd sequence length: debugging and small-scale runs
        dict(name="train_base_odd", kind="train", preset="base", layers=4, vocab=154856, batch=3, seq=777),
        # the headline benchmark's micro-batch
        dict(name="train_7b", kind="train", layers=2, batch=2, seq=4096, **wide),
        # short documents of mixed length packed into one batch, heads of 64 (0.5B preset)
        dict(name="attention_docs", kind="attention", hq=16, hk=4, d=64, tokens=8192, docs=21),
        # long-context training of the wide model: one sequence
        dict(name="attention_long", kind="attention", hq=32, hk=8, d=128, tokens=16384, docs=1),
        # four images of 1024 x 1024 in patches of 14 through one layer of the vision encoder
        dict(name="attention_images", kind="images", heads=16, d=64, tokens=5329, images=4),
        # a chat-sized prompt: time to first token
        dict(name="prefill_short", kind="prefill", layers=4, tokens=128, **wide),
        # a document-sized prompt
        dict(name="prefill_long", kind="prefill", layers=4, tokens=8192, **wide),
        # interactive decoding of one conversation
        dict(name="decode_one", kind="decode", layers=4, batch=1, context=2048, **wide),
        # the serving benchmark's batch; contexts between half and all of 4096 tokens
        dict(name="decode_batch", kind="decode", layers=4, batch=64, context=4096, **wide),
        # a few conversations over long documents
        dict(name="decode_long", kind="decode", layers=4, batch=6, context=32768, **wide),
        # the optimizer step of one layer of the wide model (138 matrices of one layer's experts and projections)
        dict(name="optimizer_7b", kind="optimizer", layers=1, **wide),
    ]


def _log(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> Dict[str, Any]:
    kind = rng.choice(["train", "train", "attention", "attention", "images", "prefill", "prefill", "decode", "decode", "decode",
                       "optimizer"])
    if kind == "train":
        preset = rng.choice(["tiny", "base", "7b"])
        layers = rng.randint(1, 2 if preset == "7b" else 4)
        tokens = _log(rng, 128, 8192)
        batch = rng.randint(1, 4)
        return dict(kind=kind, preset=preset, layers=layers, vocab=32000 if preset == "7b" else rng.choice([32000, 154856]),
                    batch=batch, seq=max(32, tokens // batch))
    if kind == "attention":
        hq, hk, d = rng.choice([(32, 8, 128), (16, 4, 64), (8, 2, 64), (16, 4, 128), (4, 2, 64)])
        tokens = _log(rng, 256, 16384)
        return dict(kind=kind, hq=hq, hk=hk, d=d, tokens=tokens, docs=rng.randint(1, max(1, min(32, tokens // 64))))
    if kind == "images":
        return dict(kind=kind, heads=rng.choice([8, 16]), d=64, tokens=_log(rng, 196, 5329), images=rng.randint(1, 4))
    wide = dict(preset="7b", vocab=32000)
    if kind == "prefill":
        return dict(kind=kind, layers=rng.randint(1, 4), tokens=_log(rng, 16, 8192), **wide)
    if kind == "decode":
        batch = _log(rng, 1, 64)
        return dict(kind=kind, layers=rng.randint(1, 4), batch=batch, context=_log(rng, 128, min(32768, 262144 // batch)), **wide)
    return dict(kind=kind, preset=rng.choice(["tiny", "base", "7b"]), layers=1, vocab=8 * _log(rng, 512, 4000))


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _config(case: Dict[str, Any]) -> YvConfig:
    if case["preset"] == "7b":
        # every layer keeps its activations, as the benchmark's planner decides on one GPU
        cfg = YvConfig.yv_7b_moe(vocab_size=case["vocab"], use_gradient_checkpointing=False)
    else:
        cfg = (YvConfig.tiny_text_moe if case["preset"] == "tiny" else YvConfig.get_base)()
        cfg.vocab_size = case["vocab"]
    cfg.n_layer = case["layers"]
    return cfg


def _model(case: Dict[str, Any], seed: int):
    """A model whose router is as decisive as a trained one: every token of the vocabulary has its experts' directions in
    its embedding, well above the rest, so that rounding does not send it elsewhere."""
    cfg = _config(case)
    model = build_model(cfg, DEV, BF16, seed=seed)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    H, E, k = cfg.hidden_size, cfg.moe_num_experts, cfg.moe_top_k
    with torch.no_grad():
        for name, p in model.named_parameters():
            if name.endswith("shared_expert_weight"):
                p.normal_(0.0, 0.5, generator=gen)
            elif p.dim() < 2:
                p.normal_(1.0, 0.1, generator=gen)
            else:          # what a branch adds to the stream is small beside the stream
                scale = 0.2 if name.endswith(("o_proj", "w2")) else 1.0
                p.normal_(0.0, scale * p.shape[-1] ** -0.5, generator=gen)
        towards = torch.linalg.qr(torch.randn(H, E, device=DEV, dtype=torch.float32, generator=gen))[0].t().contiguous()
        for layer in model.model.layers:
            layer.mlp.router.gate.weight.copy_(towards)
        embed = model.model.embed.weight.normal_(0.0, 1.0, generator=gen)
        mine = torch.rand(embed.shape[0], E, device=DEV, generator=gen).topk(k, -1).indices
        share = torch.zeros(embed.shape[0], E, device=DEV).scatter_(
            1, mine, 7.0 + 3.0 * torch.rand(mine.shape, device=DEV, generator=gen))
        embed.add_((share @ towards).to(BF16))
        if model.tied:                                  # the output head is the embedding
            model.model.norm.weight.mul_(H ** -0.5)
    return model, gen


def _ids(shape, vocab: int, gen: torch.Generator) -> torch.Tensor:
    return torch.randint(0, vocab, shape, device=DEV, generator=gen)


def _cuts(tokens: int, docs: int, seed: int) -> List[int]:
    """Offsets of ``docs`` documents of mixed length."""
    rng = random.Random(seed)
    return [0] + sorted(rng.sample(range(1, tokens), docs - 1)) + [tokens]


def _packed(case: Dict[str, Any], seed: int) -> Dict[str, Any]:
    """Queries, keys, values, gradient and sequence offsets of the two attention kinds."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    rand = lambda *shape: torch.randn(*shape, device=DEV, dtype=torch.float32, generator=gen).to(BF16)
    if case["kind"] == "attention":
        hq, hk, d, T = case["hq"], case["hk"], case["d"], case["tokens"]
        cuts = _cuts(T, case["docs"], seed)
        cos, sin = rope_tables(max(b - a for a, b in zip(cuts, cuts[1:])), d, 1e4, device=DEV)
        pos = torch.cat([torch.arange(b - a, dtype=torch.int32) for a, b in zip(cuts, cuts[1:])]).to(DEV)
        ins = dict(qkv=rand(T, (hq + 2 * hk) * d), cos=cos, sin=sin, pos=pos)
        width = hq * d
    else:
        n, T = case["images"], case["images"] * case["tokens"]
        cuts = [i * case["tokens"] for i in range(n + 1)]
        width = case["heads"] * case["d"]
        ins = dict(q=rand(T, width), k=rand(T, width), v=rand(T, width))
    return dict(ins, cuts=cuts, cu=torch.tensor(cuts, dtype=torch.int32, device=DEV), grad=rand(T, width))


def _lengths(case: Dict[str, Any], seed: int) -> List[int]:
    """Cached tokens of each sequence: between half and all of the context."""
    rng = random.Random(seed)
    return [case["context"] if i == 0 else rng.randint(case["context"] // 2, case["context"]) for i in range(case["batch"])]


def _cached(case: Dict[str, Any], cfg: YvConfig, lengths: List[int], layer: int, seed: int):
    """Keys (as rotated at their positions) and values that a layer's cache holds, packed by sequence."""
    gen = torch.Generator(device=DEV).manual_seed(seed * 64 + layer + 1)
    shape = (sum(lengths), cfg.n_kv_head, cfg.head_dim)
    return tuple(torch.randn(*shape, device=DEV, dtype=torch.float32, generator=gen).to(BF16) for _ in range(2))


def prepare(case: Dict[str, Any], seed: int) -> Dict[str, Any]:
    kind = case["kind"]
    if kind in ("attention", "images"):
        s = _packed(case, seed)
        for n in ("qkv", "q", "k", "v"):
            if n in s:
                s[n].requires_grad_(True)
        s["case"], s["longest"] = case, max(b - a for a, b in zip(s["cuts"], s["cuts"][1:]))
        return s
    model, gen = _model(case, seed)
    cfg = model.cfg
    if kind == "train":
        return dict(case=case, model=model.train(), ids=_ids((case["batch"], case["seq"]), cfg.vocab_size, gen))
    if kind == "optimizer":
        for p in model.parameters():
            p.grad = torch.randn(p.shape, device=DEV, dtype=BF16, generator=gen)
        return dict(case=case, model=model, opt=build_optimizer(model, "muon", lr=LR))
    if kind == "prefill":
        engine = YvInferenceEngine(model, cfg=YvEngineConfig(num_blocks=case["tokens"] // PAGE + 3))
        return dict(case=case, engine=engine, ids=_ids((case["tokens"],), cfg.vocab_size, gen).tolist())
    lengths = _lengths(case, seed)
    engine = YvInferenceEngine(model, cfg=YvEngineConfig(num_blocks=sum(n // PAGE + 2 for n in lengths) + 1,
                                                         graph_max_seq_len=max(8192, case["context"] + PAGE)))
    cache = engine.cache
    tokens = YvSpeculativeCacheManager(cache)
    slots = []
    for s, n in enumerate(lengths):
        cache.add_sequence(s)
        cache.append_slots(s, n)
        slots.append(torch.from_numpy(cache.slots(s, 0, n)))
        tokens.mark(s)
    slots = torch.cat(slots).to(DEV)
    for i in range(cfg.n_layer):
        for pages, rows in zip(cache.layer(i), _cached(case, cfg, lengths, i, seed)):
            pages.view(-1, cfg.n_kv_head, cfg.head_dim)[slots] = rows
    return dict(case=case, engine=engine, tokens=tokens, last=_ids((len(lengths),), cfg.vocab_size, gen).tolist())


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def _returned(name: str) -> bool:
    """All gradients but those of the one or two mixing weights of the shared experts: sums over all tokens that cancel, so
    that the rounding of sixteen-bit activations alone moves them by several percent."""
    return not name.endswith("shared_expert_weight")


def run(state: Dict[str, Any]) -> Dict[str, Any]:
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        model, ids = state["model"], state["ids"]
        model.zero_grad(set_to_none=True)
        loss = model(input_ids=ids, labels=ids, num_valid=ids.shape[0] * (ids.shape[1] - 1))["loss"]
        loss.backward()
        return dict({n: p.grad for n, p in model.named_parameters() if _returned(n)}, loss=loss.detach())
    if kind == "attention":
        # the rotation works in place on the projection that it is given: each pass has its own, as in a layer
        qkv = state["qkv"].clone()
        o = F_.rope_attention(qkv, state["cos"], state["sin"], state["pos"], state["cu"], state["longest"], case["hq"],
                              case["hk"], case["d"], case["d"])
        return {"out": o.detach(), "dqkv": torch.autograd.grad(o, state["qkv"], state["grad"])[0]}
    if kind == "images":
        ins = [state[n] for n in "qkv"]
        o = F_.attention(*ins, state["cu"], state["cu"], state["longest"], state["longest"], case["heads"], case["heads"],
                         case["d"])
        grads = torch.autograd.grad(o, ins, state["grad"])
        return dict(zip(("dq", "dk", "dv"), grads), out=o.detach())
    if kind == "optimizer":
        state["opt"].step()
        return {n: p.detach() for n, p in state["model"].named_parameters()}
    engine = state["engine"]
    if kind == "prefill":
        engine.cache.add_sequence(0)
        logits = engine.run_tokens(0, state["ids"], [len(state["ids"]) - 1])
        engine.cache.free_sequence(0)
        return {"logits": logits, "k": engine.cache.k, "v": engine.cache.v}
    seqs = list(range(case["batch"]))
    logits = engine.graph.step(state["last"], seqs)
    for s in seqs:
        state["tokens"].rollback(s, 0)
    return {"logits": logits}


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _sizes(cfg: YvConfig) -> Dict[str, float]:
    """Parameters of a layer: attention, one routed expert, shared experts, router."""
    H = cfg.hidden_size
    F, Fs = cfg.moe_expert_intermediate_size, cfg.moe_shared_intermediate_size
    return {"attention": H * (2 * cfg.n_head + 2 * cfg.n_kv_head) * cfg.head_dim, "expert": 3 * H * F,
            "shared": 3 * H * Fs * cfg.moe_shared_experts, "router": H * cfg.moe_num_experts}


def _seen(lengths: List[int], causal: bool) -> float:
    """Pairs of a query and a key."""
    return float(sum(n * (n + 1) / 2 if causal else n * n for n in lengths))


def work(case: Dict[str, Any]) -> Dict[str, float]:
    kind = case["kind"]
    if kind in ("attention", "images"):
        if kind == "attention":
            hq, hk, d, T = case["hq"], case["hk"], case["d"], case["tokens"]
            cuts = _cuts(T, case["docs"], 0)
            lengths = [b - a for a, b in zip(cuts, cuts[1:])]
        else:
            hq = hk = case["heads"]
            d, T, lengths = case["d"], case["images"] * case["tokens"], [case["tokens"]] * case["images"]
        # two products forward, five backward; q, k, v, the output and its gradient are read, output and gradients written
        return {"flops": 14.0 * hq * d * _seen(lengths, kind == "attention"),
                "bytes": 2.0 * T * d * (2 * (hq + 2 * hk) + 2 * hq)}
    cfg = _config(case)
    H, L, V, E, k = cfg.hidden_size, cfg.n_layer, cfg.vocab_size, cfg.moe_num_experts, cfg.moe_top_k
    z = _sizes(cfg)
    dense = z["attention"] + z["shared"] + z["router"]
    if kind == "optimizer":
        # ten iterations of three products on the short side of each matrix, symmetric ones at half
        flops = 0.0
        F, Fs, S, nq, nk = (cfg.moe_expert_intermediate_size, cfg.moe_shared_intermediate_size, cfg.moe_shared_experts,
                            cfg.n_head * cfg.head_dim, cfg.n_kv_head * cfg.head_dim)
        for count, n, m in ((2 * E, F, H), (E, H, F), (2 * S, Fs, H), (1, H, S * Fs), (1, nq, H), (2, nk, H), (1, H, nq)):
            a, b = min(n, m), max(n, m)
            flops += count * 10.0 * (2.0 * a * a * b + a * a * b + a * a * a)
        params = dense + E * z["expert"] + V * H * (1 if cfg.tie_word_embeddings else 2)
        return {"flops": L * flops, "bytes": 2.0 * params * 5}
    if kind == "train":
        T = case["batch"] * case["seq"]
        params = L * (dense + E * z["expert"]) + V * H
        flops = 6.0 * T * (L * (dense + k * z["expert"]) + V * H)
        flops += 12.0 * L * cfg.n_head * cfg.head_dim * _seen([case["seq"]] * case["batch"], True)
        return {"flops": flops, "bytes": 2.0 * 2 * params}
    if kind == "prefill":
        T, context = case["tokens"], case["tokens"] * (case["tokens"] + 1) / 2
        read = 0.0
        rows = 1
    else:
        lengths = _lengths(case, 0)
        T, context, read = case["batch"], float(sum(lengths)), float(sum(lengths))
        rows = T
    experts = E * (1 - (1 - k / E) ** T)          # experts that some token is sent to
    kv = 2.0 * cfg.n_kv_head * cfg.head_dim
    return {"flops": 2.0 * T * L * (dense + k * z["expert"]) + 2.0 * rows * V * H + 4.0 * L * cfg.n_head * cfg.head_dim * context,
            "bytes": 2.0 * (L * (dense + experts * z["expert"] + kv * (read + T)) + V * H + T * H) + 4.0 * rows * V}


def tolerance(case: Dict[str, Any]) -> Any:
    """About four times the distance from 64 bits that was measured over the ranges: sixteen-bit weights, activations and
    probabilities (outputs of attention 0.003, its gradients 0.005 to 0.013, logits 0.006, a model's gradients 0.005 to 0.01),
    and weights that are rounded to 16 bits after the step (0.002)."""
    return {"rel": 0.01, "max": 0.4} if case["kind"] == "optimizer" else {"rel": 0.03, "max": 0.9}


# ------------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------------
class _Attention64(torch.autograd.Function):
    """Softmax attention of packed sequences, q [Tq, hq, d] over k, v [Tk, hk, d], in pieces of 1024 queries; with ``causal``
    the last query of a sequence sees all of its keys."""

    @staticmethod
    def pieces(cq: List[int], ck: List[int]):
        for b in range(len(cq) - 1):
            for lo in range(cq[b], cq[b + 1], 1024):
                yield b, lo, min(lo + 1024, cq[b + 1])

    @staticmethod
    def weights(q, k, b, lo, hi, cq, ck, causal):
        hk = k.shape[1]
        end = ck[b + 1] - (cq[b + 1] - hi) if causal else ck[b + 1]
        qs = q[lo:hi].reshape(hi - lo, hk, -1, q.shape[2])
        s = torch.einsum("qhgd,khd->hgqk", qs, k[ck[b]:end]) * q.shape[2] ** -0.5
        if causal:
            at = torch.arange(hi - lo, device=q.device) + (end - ck[b]) - (hi - lo)
            s.masked_fill_(torch.arange(end - ck[b], device=q.device)[None, :] > at[:, None], float("-inf"))
        return qs, slice(ck[b], end), torch.softmax(s, -1)

    @staticmethod
    def forward(ctx, q, k, v, cq, ck, causal):
        ctx.save_for_backward(q, k, v)
        ctx.rest = (cq, ck, causal)
        out = torch.empty_like(q)
        for b, lo, hi in _Attention64.pieces(cq, ck):
            _, keys, p = _Attention64.weights(q, k, b, lo, hi, cq, ck, causal)
            out[lo:hi] = torch.einsum("hgqk,khd->qhgd", p, v[keys]).reshape(hi - lo, q.shape[1], -1)
        return out

    @staticmethod
    def backward(ctx, grad):
        q, k, v = ctx.saved_tensors
        cq, ck, causal = ctx.rest
        dq, dk, dv = torch.empty_like(q), torch.zeros_like(k), torch.zeros_like(v)
        for b, lo, hi in _Attention64.pieces(cq, ck):
            qs, keys, p = _Attention64.weights(q, k, b, lo, hi, cq, ck, causal)
            g = grad[lo:hi].reshape(hi - lo, k.shape[1], -1, v.shape[2])
            dv[keys] += torch.einsum("hgqk,qhgd->khd", p, g)
            dp = torch.einsum("qhgd,khd->hgqk", g, v[keys])
            ds = p * (dp - (dp * p).sum(-1, keepdim=True)) * q.shape[2] ** -0.5
            dq[lo:hi] = torch.einsum("hgqk,khd->qhgd", ds, k[keys]).reshape(hi - lo, q.shape[1], -1)
            dk[keys] += torch.einsum("hgqk,qhgd->khd", ds, qs)
        return dq, dk, dv, None, None, None


def _rotate64(x: torch.Tensor, pos: torch.Tensor, theta: float) -> torch.Tensor:
    half = x.shape[2] // 2
    angle = pos.double()[:, None, None] * theta ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    c, s, a, b = angle.cos(), angle.sin(), x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _norm64(x: torch.Tensor, w: torch.Tensor, eps: float) -> torch.Tensor:
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _ffn64(x: torch.Tensor, w13: torch.Tensor, w2: torch.Tensor, scale: Any = 1.0) -> torch.Tensor:
    gate, up = (x @ w13.t()).chunk(2, -1)
    return (torch.nn.functional.silu(gate) * up * scale) @ w2.t()


def _experts64(x: torch.Tensor, w: Dict[str, torch.Tensor], p: str, cfg: YvConfig) -> torch.Tensor:
    prob = torch.softmax(x @ w[p + "router.gate.weight"].t(), -1)
    top, idx = prob.topk(cfg.moe_top_k, -1)
    top = top / top.sum(-1, keepdim=True)
    S, out = cfg.moe_shared_experts, torch.zeros_like(x)
    mix = torch.softmax(w[p + "shared_expert_weight"], 0)
    w13, w2 = w[p + "shared_w13"].chunk(S, 0), w[p + "shared_w2"].chunk(S, 1)
    for s in range(S):
        out = out + _ffn64(x, w13[s], w2[s], mix[s])
    for e in range(cfg.moe_num_experts):
        token, place = (idx == e).nonzero(as_tuple=True)
        if token.numel():
            y = _ffn64(x[token], w[p + "experts_w13"][e], w[p + "experts_w2"][e], top[token, place][:, None])
            out = out.index_add(0, token, y)
    return out


def _trunk64(w: Dict[str, torch.Tensor], cfg: YvConfig, ids: torch.Tensor, pos: torch.Tensor, cq: List[int], ck: List[int],
             cached=None) -> torch.Tensor:
    """Final hidden states of the tokens; ``cached(layer)`` are keys and values in front of each sequence's own."""
    hq, hk, d = cfg.n_head, cfg.n_kv_head, cfg.head_dim
    h = w["model.embed.weight"][ids]
    for i in range(cfg.n_layer):
        p = f"model.layers.{i}."
        qkv = (_norm64(h, w[p + "norm_attention.weight"], cfg.layer_norm_eps) @ w[p + "attention.qkv_proj"].t())
        q, k, v = (t.view(-1, n, d) for t, n in zip(qkv.split([hq * d, hk * d, hk * d], 1), (hq, hk, hk)))
        q, k = _rotate64(q, pos, cfg.rope_theta), _rotate64(k, pos, cfg.rope_theta)
        if cached is not None:
            old, lens = cached(i), [b - a for a, b in zip(ck, ck[1:])]
            k, v = (torch.cat([t for a, b in zip(o.double().split([n - 1 for n in lens]), new.split(1)) for t in (a, b)])
                    for o, new in zip(old, (k, v)))
        h = h + _Attention64.apply(q, k, v, cq, ck, True).reshape(-1, hq * d) @ w[p + "attention.o_proj"].t()
        h = h + _experts64(_norm64(h, w[p + "norm_mlp.weight"], cfg.layer_norm_eps), w, p + "mlp.", cfg)
    return _norm64(h, w["model.norm.weight"], cfg.layer_norm_eps)


def _orthogonal64(x: torch.Tensor) -> torch.Tensor:
    x = x / x.norm(dim=(1, 2), keepdim=True)
    flip = x.shape[1] > x.shape[2]
    x = x.transpose(1, 2) if flip else x
    eye = torch.eye(x.shape[1], device=x.device, dtype=x.dtype)
    for a, b, c in NS_COEFFS:
        g = x @ x.transpose(1, 2)
        x = (a * eye + b * g + c * (g @ g)) @ x
    return x.transpose(1, 2) if flip else x


def _muon64(name: str, p: torch.Tensor, g: torch.Tensor, cfg: YvConfig) -> torch.Tensor:
    """The matrices that a parameter stacks, each moved along its orthogonalised gradient (first step: the momentum is the
    gradient)."""
    d, H = cfg.head_dim, cfg.hidden_size
    if name.endswith("qkv_proj"):
        rows = [cfg.n_head * d] + 2 * [cfg.n_kv_head * d]
        parts = list(zip(p.split(rows), g.split(rows)))
    elif name.endswith(("experts_w13", "shared_w13")):
        rows = cfg.moe_expert_intermediate_size if "experts" in name else cfg.moe_shared_intermediate_size
        parts = [(p.reshape(-1, rows, H), g.reshape(-1, rows, H))]
    else:
        parts = [(p, g)]
    out = []
    for t, u in parts:
        t3, u3 = t.reshape(-1, *t.shape[-2:]), u.reshape(-1, *u.shape[-2:])
        n, m = t3.shape[1:]
        step = LR * 0.18 * math.sqrt(max(n, m) / min(n, m))
        out += [(a.double() * (1 - LR * 0.1) - step * _orthogonal64(b.double()[None])[0]).float() for a, b in zip(t3, u3)]
    return torch.cat([o.reshape(-1) for o in out]).view(p.shape).double()


def exact(case: Dict[str, Any], seed: int) -> Optional[Dict[str, Any]]:
    kind = case["kind"]
    if kind == "attention":
        s = _packed(case, seed)
        hq, hk, d = case["hq"], case["hk"], case["d"]
        qkv = s["qkv"].double().requires_grad_(True)
        q, k, v = (t.view(-1, n, d) for t, n in zip(qkv.split([hq * d, hk * d, hk * d], 1), (hq, hk, hk)))
        q, k = _rotate64(q, s["pos"], 1e4), _rotate64(k, s["pos"], 1e4)
        o = _Attention64.apply(q, k, v, s["cuts"], s["cuts"], True).reshape(-1, hq * d)
        return {"out": o.detach(), "dqkv": torch.autograd.grad(o, qkv, s["grad"].double())[0]}
    if kind == "images":
        s = _packed(case, seed)
        ins = [s[n].double().requires_grad_(True) for n in "qkv"]
        o = _Attention64.apply(*(t.view(-1, case["heads"], case["d"]) for t in ins), s["cuts"], s["cuts"], False)
        o = o.reshape(ins[0].shape)
        return dict(zip(("dq", "dk", "dv"), torch.autograd.grad(o, ins, s["grad"].double())), out=o.detach())
    if kind == "optimizer":
        s = prepare(case, seed)
        cfg = s["model"].cfg
        out = {}
        for n, p in s["model"].named_parameters():
            if s["opt"].is_muon_param(n, p):
                out[n] = _muon64(n, p.detach(), p.grad, cfg)
            else:         # AdamW's first step: the sign of the gradient, but for the added epsilon
                g = p.grad.double()
                out[n] = p.detach().double() * (1 - LR * 0.1) - LR * g / (g.abs() + 1e-8)
        return out
    model, gen = _model(case, seed)
    cfg = model.cfg
    w = {n: p.detach().double() for n, p in model.named_parameters()}
    head = "model.embed.weight" if model.tied else "lm_head"
    if kind == "train":
        ids = _ids((case["batch"], case["seq"]), cfg.vocab_size, gen)
        B, S = ids.shape
        del model
        for t in w.values():
            t.requires_grad_(True)
        cuts = [i * S for i in range(B + 1)]
        h = _trunk64(w, cfg, ids.reshape(-1), torch.arange(S, device=DEV).repeat(B), cuts, cuts)
        h, want = h.view(B, S, -1)[:, :-1].reshape(B * (S - 1), -1), ids[:, 1:].reshape(-1)
        # the loss's gradient at the final states, some rows at a time
        leaf, rows = h.detach().requires_grad_(True), 1024
        for lo in range(0, want.numel(), rows):
            logits = leaf[lo:lo + rows] @ w[head].t()
            part = torch.nn.functional.cross_entropy(logits, want[lo:lo + rows], reduction="sum") / want.numel()
            part.backward()
        h.backward(leaf.grad)
        # the loss itself is a mean in which the roundings of thousands of tokens cancel: how far it is off is chance
        return dict({n: t.grad for n, t in w.items() if _returned(n)}, loss=None)
    with torch.no_grad():
        if kind == "prefill":
            n = case["tokens"]
            ids = _ids((n,), cfg.vocab_size, gen)
            h = _trunk64(w, cfg, ids, torch.arange(n, device=DEV), [0, n], [0, n])
            none = [None] * cfg.n_layer
            return {"logits": h[-1:] @ w[head].t(), "k": none, "v": none}
        lengths = _lengths(case, seed)
        ids = _ids((len(lengths),), cfg.vocab_size, gen)
        ck = [0]
        for n in lengths:
            ck.append(ck[-1] + n + 1)
        h = _trunk64(w, cfg, ids, torch.tensor(lengths, device=DEV), list(range(len(lengths) + 1)), ck,
                     lambda i: _cached(case, cfg, lengths, i, seed))
        return {"logits": h @ w[head].t()}
