"""Mixture-of-experts operators: routing (gate kernel), and the routed expert computation
(permute -> grouped GEMM -> SwiGLU -> grouped GEMM -> weighted combine) as one autograd function that
never synchronises with the host: the expert-sorted row buffer is sized by its upper bound
``T*k + E*127`` and the grouped GEMM reads the real tile count from device memory.

Replaces the reference's Python expert loop (model/moe/layer.py:915-936) and its "fused" dispatch with a
``.cpu().tolist()`` sync (opss/infer/fused_moe.py:54-123).
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch
from torch.utils.weak import WeakIdKeyDictionary

from . import kernels, reference as ref, status_word

_BF16 = torch.bfloat16


def _k():
    return kernels()


# --------------------------------------------------------------------------------------------------
# routing
# --------------------------------------------------------------------------------------------------
def gate_topk(logits: torch.Tensor, bias: Optional[torch.Tensor], k: int, bias_in_combine: bool = True,
              renorm_mode: int = 0) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor]:
    """logits [T,E] -> (weights [T,k] fp32, idx [T,k], counts [E], probs [T,E]).

    ``bias`` (aux-loss-free balancing) is added before the softmax when ``bias_in_combine`` (reference
    behaviour, model/moe/gate.py:378) or only to the selection key otherwise (DeepSeek-V3 style).
    ``renorm_mode`` 0 divides the selected probabilities by their sum; 1 applies a softmax over them
    (reference, gate.py:1221)."""
    if logits.is_cuda:
        b = bias.float().contiguous() if bias is not None else None
        return _k().route(logits, b, k, bias_in_combine, renorm_mode)
    w, idx, probs, counts = ref.gate_topk(logits, bias, k, bias_in_combine, renorm_mode)
    return w, idx, counts, probs


_PLAN_TOKENS = 16        # kPlanTokens of csrc/yv_ops.h


def route_few(logits: torch.Tensor, bias: Optional[torch.Tensor], k: int, bias_in_combine: bool = True, renorm_mode: int = 0):
    """``gate_topk`` of a few tokens without a gradient, and the experts' dispatch plan, in one kernel: (weights, idx, counts,
    plan, a zero on the device), or None where that does not apply."""
    if not logits.is_cuda or torch.is_grad_enabled() or not 1 <= logits.shape[0] <= _PLAN_TOKENS or logits.shape[1] > 256 or \
            logits.dtype != torch.float32 or not logits.is_contiguous() or not 1 <= k <= 16:
        return None
    return _k().route_few(logits, None if bias is None else bias.float().contiguous(), k, bias_in_combine, renorm_mode)


# --------------------------------------------------------------------------------------------------
# dispatch plan
# --------------------------------------------------------------------------------------------------
class DispatchPlan:
    """Device-side description of one expert-sorted, 128-row-padded token layout."""
    __slots__ = ("seg_offsets", "tile_expert", "num_m_tiles", "row_map", "counts", "max_rows", "k")

    def __init__(self, seg_offsets, tile_expert, num_m_tiles, row_map, counts, max_rows, k):
        self.seg_offsets, self.tile_expert, self.num_m_tiles = seg_offsets, tile_expert, num_m_tiles
        self.row_map, self.counts, self.max_rows, self.k = row_map, counts, max_rows, k


def padded_rows_bound(num_assignments: int, num_experts: int) -> int:
    """Upper bound of the padded row count: every expert wastes at most 127 rows."""
    return ((num_assignments + num_experts * 127 + 127) // 128) * 128


def permute_tokens(x: torch.Tensor, idx: torch.Tensor, counts: torch.Tensor, num_experts: int,
                   deterministic: bool = False, zero_pad: bool = True) -> Tuple[torch.Tensor, DispatchPlan]:
    """Scatter token rows into expert-sorted order.  Returns (xp [max_rows, H], plan).  The pad rows of every expert
    segment are zeroed unless ``zero_pad`` is off: the weight-gradient GEMMs sum over whole segments, so training
    needs zeros there; inference never reads what the pad rows produce."""
    T, H = x.shape
    k = idx.shape[1]
    dev = x.device
    max_rows = padded_rows_bound(T * k, num_experts)
    K = _k()
    seg = torch.empty(num_experts + 1, dtype=torch.int32, device=dev)
    tile_expert = torch.empty(max_rows // 128, dtype=torch.int32, device=dev)
    num_tiles = torch.empty(1, dtype=torch.int32, device=dev)
    cursor = torch.empty(num_experts, dtype=torch.int32, device=dev)
    K.moe_plan(counts, seg, tile_expert, num_tiles, cursor)
    xp = torch.empty(max_rows, H, dtype=_BF16, device=dev)
    row_map = torch.empty(T, k, dtype=torch.int32, device=dev)
    if deterministic:
        # assignment order inside an expert follows token order (what a stable sort by expert would give): one CTA per
        # expert counts its assignments in order
        K.moe_rank(idx.contiguous(), seg, row_map)
        K.moe_permute(x, idx, None, row_map, xp)
    else:
        K.moe_permute(x, idx, cursor, row_map, xp)
    if zero_pad:
        K.moe_zero_pad(xp, seg, counts)
    return xp, DispatchPlan(seg, tile_expert, num_tiles, row_map, counts, max_rows, k)


def _few_tokens(assignments: int, w13: torch.Tensor, w2: torch.Tensor) -> bool:
    """Whether the experts' weights are read for so few tokens that reading them is most of the time there is.  64 experts
    of 4096 x 1408, both products and the activation, top-6 of T tokens, us: T = 64 435 by the general kernel and 350 by
    this one, 1024 434 and 373, 1536 578 and 492, 2048 (192 tokens an expert) 585 and 525, 3072 847 and 889.  A whole layer of 8
    experts of 256 x 256, top-2: T = 1 48 and 35, 512 50 and 47; of 16 of 1024 x 704, top-2: T = 1 73 and 40, 1024 104 and 90."""
    E, F = w2.shape[0], w2.shape[2]
    return assignments <= 192 * E and F % 64 == 0 and w13.is_contiguous() and w2.is_contiguous()


def _few_slots(tokens: int, k: int, E: int) -> int:
    """Token slots per pass over a tile's weights: no expert gets a token twice from the router, and a second pass (80 % of the
    first one's time again at T = 1024) costs far more than empty slots (1 us)."""
    return min(tokens, 64 if tokens * k <= 16 * E else 128)


class _MxExpertsFn(torch.autograd.Function):
    """Routed experts whose forward products run on the block-scaled fp8 tensor cores: rows quantised per 32 elements on the fly,
    the expert weights once per optimizer step; backward stays in bf16 from the saved bf16 tensors, which are those of the
    function in ``csrc/binding_autograd.inc``."""

    @staticmethod
    def forward(ctx, x, w13, w2, weights, idx, counts, deterministic, add):
        from ..quant import fp8 as q8
        K = _k()
        st = status_word(x.device)
        T, H = x.shape
        E, twoF, _ = w13.shape
        F = twoF // 2
        x = x.contiguous()
        add = None if add is None else add.contiguous()
        xp, plan = permute_tokens(x, idx, counts, E, deterministic, zero_pad=True)
        wts = weights.float().contiguous()
        y1 = torch.empty(plan.max_rows, twoF, dtype=_BF16, device=x.device)
        act = torch.empty(plan.max_rows, F, dtype=_BF16, device=x.device)
        y2 = torch.empty(plan.max_rows, H, dtype=_BF16, device=x.device)
        xq, xs = q8.quantize_mx(xp)
        del xp
        wq, ws = _mx_weight(w13)
        K.gemm_mxfp8(xq, xs, wq, ws, y1, plan.tile_expert, plan.num_m_tiles, 0, st)
        del xq, xs
        K.swiglu_fwd(y1, act)
        aq, as_ = q8.quantize_mx(act)
        wq, ws = _mx_weight(w2)
        K.gemm_mxfp8(aq, as_, wq, ws, y2, plan.tile_expert, plan.num_m_tiles, 0, st)
        del aq, as_, act
        out = torch.empty(T, H, dtype=_BF16, device=x.device)
        K.moe_combine(y2, plan.row_map, wts, add, out)
        ctx.save_for_backward(x, y1, w13, w2, wts, idx, plan.row_map, plan.seg_offsets, plan.tile_expert,
                              plan.num_m_tiles, plan.counts)
        ctx.dims = (T, H, E, F, plan.max_rows, idx.shape[1])
        ctx.w_dtype = weights.dtype
        ctx.has_add = add is not None
        return out

    @staticmethod
    def backward(ctx, dout):
        K = _k()
        x, y1, w13, w2, wts, idx, row_map, seg, tile_expert, num_tiles, counts = ctx.saved_tensors
        T, H, E, F, max_rows, k = ctx.dims
        st = status_word(dout.device)
        dev = dout.device
        dout = dout.contiguous()
        # combine weight of every expert row (0 on pad rows)
        row_w = torch.zeros(max_rows, dtype=torch.float32, device=dev)
        K.moe_row_weights(wts, row_map, row_w)
        # unweighted output gradient in expert-row order
        dy2 = torch.empty(max_rows, H, dtype=_BF16, device=dev)
        K.moe_permute(dout, idx, None, row_map, dy2)
        K.moe_zero_pad(dy2, seg, counts)
        # down projection (unweighted activation gradient), then the activation with the weights applied
        dact = torch.empty(max_rows, F, dtype=_BF16, device=dev)
        K.gemm_grouped_m(dy2, w2, dact, tile_expert, num_tiles, True, 0, st)          # dy2 [rows,H] x w2[e] [H,F]
        dy1 = torch.empty_like(y1)
        act_w = torch.empty(max_rows, F, dtype=_BF16, device=dev)
        rowdot = torch.empty(max_rows, dtype=torch.float32, device=dev)
        K.swiglu_bwd_rows(y1, dact, row_w, dy1, act_w, rowdot)
        del dact
        dw2 = torch.empty_like(w2)
        K.gemm_grouped_k(dy2, act_w, dw2, seg, False, 0, st)                          # [H, rows_e] x [rows_e, F]
        del dy2, act_w
        dwts = torch.empty(T, k, dtype=torch.float32, device=dev)
        K.moe_row_dots(rowdot, row_map, dwts)
        # up projection
        dxp = torch.empty(max_rows, H, dtype=_BF16, device=dev)
        K.gemm_grouped_m(dy1, w13, dxp, tile_expert, num_tiles, True, 0, st)          # dy1 [rows,2F] x w13[e] [2F,H]
        xp = torch.empty(max_rows, H, dtype=_BF16, device=dev)
        K.moe_permute(x, idx, None, row_map, xp)
        K.moe_zero_pad(xp, seg, counts)
        dw13 = torch.empty_like(w13)
        K.gemm_grouped_k(dy1, xp, dw13, seg, False, 0, st)
        del xp, dy1
        dx = torch.empty(T, H, dtype=_BF16, device=dev)
        K.moe_unpermute_sum(dxp, row_map, dx, k)
        return dx, dw13, dw2, dwts.to(ctx.w_dtype), None, None, None, (dout if ctx.has_add else None)


_MX_WEIGHTS = WeakIdKeyDictionary()      # the copies of a weight live as long as the tensor that they were made of


def _mx_weight(w: torch.Tensor):
    """Block-scaled copy of a stacked expert weight [E, N, K] (quantised again only after the tensor changed)."""
    from ..quant import fp8 as q8
    key = (w.data_ptr(), w._version, tuple(w.shape))
    hit = _MX_WEIGHTS.get(w)
    if hit is None or hit[0] != key:
        E, N, Kd = w.shape
        q, sf = q8.quantize_mx(w.detach().reshape(E * N, Kd))
        hit = (key, q.view(E, N, Kd), sf)
        _MX_WEIGHTS[w] = hit
    return hit[1], hit[2]


def moe_experts(x: torch.Tensor, w13: torch.Tensor, w2: torch.Tensor, weights: torch.Tensor, idx: torch.Tensor,
                counts: Optional[torch.Tensor] = None, deterministic: bool = False,
                fp8: Optional[str] = None, add: Optional[torch.Tensor] = None, few: bool = True,
                plan: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Routed experts: out[t] = sum_j weights[t,j] * SwiGLU_FFN_{idx[t,j]}(x[t]).

    x [T,H]; w13 [E, 2F, H] (gate rows then up rows); w2 [E, H, F]; weights/idx [T,k]; counts [E] int32
    (the histogram the gate kernel produced; recomputed when omitted).  ``fp8="mx"`` runs the two forward products
    with e4m3 operands and one power-of-two scale per 32 elements (CUDA; H, F multiples of 128).  ``add`` [T,H], the shared
    experts' output, is added before the result is rounded.  ``few`` lets a pass without a gradient take the kernel for few
    tokens, which rounds in other places; off, it equals a pass with a gradient bit for bit.  ``plan``: what ``route_few`` returned with
    these ``idx``."""
    if not x.is_cuda:
        out = ref.moe_experts(x, w13, w2, weights, idx)
        return out if add is None else out + add
    E = w13.shape[0]
    if counts is None:
        counts = torch.bincount(idx.flatten().long(), minlength=E).int()
    x, idx, counts = x.to(_BF16), idx.int(), counts.int()
    add = None if add is None else add.to(_BF16)
    training = torch.is_grad_enabled()
    F, H = w13.shape[1] // 2, x.shape[1]
    if fp8 == "mx" and H % 128 == 0 and F % 128 == 0:
        return _MxExpertsFn.apply(x, w13, w2, weights, idx, counts, deterministic, add)
    # without autograd (inference) nothing reads what the pad rows of the expert segments produce: zeroing them is skipped
    T, k = idx.shape
    slots = _few_slots(T, k, E) if few and not training and _few_tokens(T * k, w13, w2) else 0
    return _k().moe_experts(x, w13, w2, weights, add, idx, counts, None if deterministic else plan, deterministic, training, slots,
                            status_word(x.device))


def capacity_mask(weights: torch.Tensor, idx: torch.Tensor, probs: torch.Tensor, counts: torch.Tensor,
                  capacity: int) -> torch.Tensor:
    """Capacity rule on the GPU: inside every expert keep the ``capacity`` assignments with the highest routing
    probability (ties by token order), zero the others and renormalise each token's weights.  No autograd: the
    result replaces the gate's weights in the forward value, gradients flow through the kept weights' own graph in
    the caller."""
    keep = torch.empty(idx.shape, dtype=torch.uint8, device=idx.device)
    out = torch.empty(idx.shape, dtype=torch.float32, device=idx.device)
    _k().moe_capacity_mask(weights.detach().float().contiguous(), idx.int().contiguous(), probs.detach().float().contiguous(),
                           counts.int().contiguous(), keep, out, int(capacity))
    return out, keep


def update_gate_bias(bias: torch.Tensor, counts: torch.Tensor, rate: float, clamp: float = 2.0) -> None:
    """Aux-loss-free balancing: bias += rate * (1/E - usage), clamped (reference gate.py:1059-1094)."""
    if bias.is_cuda:
        _k().gate_bias_update(bias, counts.int(), rate, clamp)
        return
    usage = counts.float() / counts.sum().clamp_min(1).float()
    bias.add_(rate * (1.0 / bias.numel() - usage)).clamp_(-clamp, clamp)
