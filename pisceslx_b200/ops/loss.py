"""Fused LM-head + cross-entropy: logits are produced chunk by chunk ([chunk, V] fp32), turned into
per-token losses and logit gradients by one kernel, and immediately contracted into dH and dW, so that
logits of many rows never exist at once (the reference materialises [T, V], model/core/model.py:2440,2505);
``rows_at_once`` says how many rows a chunk holds.
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from . import kernels, reference as ref, status_word

_BF16 = torch.bfloat16


def _slices(M: int, N: int, K: int) -> int:
    """Slices of K for the gradient of the hidden states, [M, V] x [V, N]: a long sum over few output tiles.

    Counted in steps of 64 by all SMs (0.45 us each for a 128 x 256 tile) and in bytes of the fp32 parts, which are written and
    read (5 TB/s); one slice unless that saves a fifth.  At 154856 x 1024: 2048 rows 670 us in one slice, 517 in nine; 283 rows
    679 and 108 (twelve)."""
    tiles, steps = -(-M // 128) * -(-N // 256), -(-K // 64)
    if tiles > 148 or steps < 64 or N % 4:
        return 1

    def cost(s: int) -> float:
        return 0.45 * -(-tiles * s // 148) * -(-steps // s) + (M * N * 8e-6 * s / 5 + 5 if s > 1 else 0)

    best = min(range(1, 17), key=cost)
    return best if cost(best) < 0.8 * cost(1) else 1


def _times_weights(dl: torch.Tensor, w: torch.Tensor, out: torch.Tensor, st: torch.Tensor) -> None:
    """out [n, H] = dl [n, V] @ w [V, H]."""
    (M, K), N = dl.shape, w.shape[1]
    s = _slices(M, N, K)
    if s == 1:
        kernels().gemm(dl, w, out, False, True, False, 0, st)
        return
    per = -(-(-(-K // 64)) // s) * 64
    cuts = torch.arange(0, (s + 1) * per, per, dtype=torch.int32, device=dl.device).clamp_(max=K)
    parts = torch.empty(s, -(-M // 128) * 128, N, dtype=torch.float32, device=dl.device)
    kernels().gemm_split(dl, w, parts, cuts, out, st)


class _LinearCEFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, h, w, labels, ignore_index, scale, chunk):
        K = kernels()
        st = status_word(h.device)
        T, H = h.shape
        V = w.shape[0]
        dev = h.device
        h = h.contiguous()
        need_dh = ctx.needs_input_grad[0]
        need_dw = ctx.needs_input_grad[1]
        loss_rows = torch.empty(T, dtype=torch.float32, device=dev)
        dh = torch.empty_like(h) if need_dh else None
        n_chunks = -(-T // max(chunk, 1))
        dw32 = None
        dw = None
        if need_dw:
            if n_chunks > 1:
                dw32 = torch.zeros(V, H, dtype=torch.float32, device=dev)
            else:
                dw = torch.empty(V, H, dtype=_BF16, device=dev)
        logits = torch.empty(min(chunk, T), V, dtype=torch.float32, device=dev)
        dlogits = torch.empty(min(chunk, T), V, dtype=_BF16, device=dev) if (need_dh or need_dw) else None
        for c in range(n_chunks):
            r0, r1 = c * chunk, min(T, (c + 1) * chunk)
            n = r1 - r0
            lg = logits[:n]
            K.gemm(h[r0:r1], w, lg, False, False, False, 0, st)
            dl = dlogits[:n] if dlogits is not None else None
            K.ce_fwd_bwd(lg, labels[r0:r1], loss_rows[r0:r1], dl, ignore_index, scale)
            if need_dh:
                _times_weights(dl, w, dh[r0:r1], st)
            if need_dw:
                if dw32 is not None:
                    K.gemm(dl, h[r0:r1], dw32, True, True, True, 0, st)             # [V,n] x [n,H], accumulate
                else:
                    K.gemm(dl, h[r0:r1], dw, True, True, False, 0, st)
        if dw32 is not None:
            dw = dw32.to(_BF16)
            del dw32
        ctx.save_for_backward(dh, dw)
        return loss_rows.sum() * scale

    @staticmethod
    def backward(ctx, gout):
        dh, dw = ctx.saved_tensors
        K = kernels()
        g = gout.reshape(1).float().contiguous()
        if dh is not None:
            K.scale_(dh, g, 1.0)
        if dw is not None:
            K.scale_(dw, g, 1.0)
        return dh, dw, None, None, None, None


_ONE_CHUNK = 2 << 30     # bytes: 1.2 % of the card's memory


def rows_at_once(T: int, V: int, H: int, chunk: int = 2048, weight_grad: bool = True) -> int:
    """Rows of logits to hold at a time.  One chunk saves the fp32 sum of the weight gradient that several add to: its zeros, its
    reads and writes by every chunk and its conversion.  Head and loss of 2331 rows of 1024, 154856 words, 3035 us in two chunks
    and 2566 in one; of 8192 rows of 4096, 32000 words, 6207 in four and 5231.  So all rows are held where the weight gradient is
    wanted and they, in fp32 and with their gradient in bf16, take no more than several chunks and that sum (the first of these
    two: 2.2 GB for 2.5), or at most 2 GB (the second: 1.57 GB, where four chunks and the sum take 0.92)."""
    one = 6 * T * V
    return T if T <= chunk or weight_grad and one <= max(6 * chunk * V + 4 * V * H, _ONE_CHUNK) else chunk


def linear_cross_entropy(h: torch.Tensor, w: torch.Tensor, labels: torch.Tensor, ignore_index: int = -100,
                         num_valid: Optional[int] = None, chunk: int = 2048) -> torch.Tensor:
    """Mean next-token loss of ``softmax(h @ w.T)`` against ``labels`` (already shifted by the caller).

    h [T,H], w [V,H], labels [T] int64.  ``num_valid`` is the number of labels != ignore_index; pass it
    from the host-side batch to avoid a device synchronisation (it is counted on the device otherwise)."""
    if num_valid is None:
        num_valid = int((labels != ignore_index).sum().item())
    scale = 1.0 / max(num_valid, 1)
    if h.is_cuda:
        return _LinearCEFn.apply(h.to(_BF16), w, labels.contiguous(), ignore_index, scale, chunk)
    loss, _ = ref.linear_cross_entropy(h, w, labels, ignore_index)
    return loss * scale
