"""Front-end of the tcgen05 flash-attention forward kernel (``csrc/attention.cu``).

``flash_attention`` takes query/key/value in the ``[batch, time, heads, head_dim]`` layout of the attention layers.  The
forward pass runs on this package's kernel; the backward pass recomputes the attention through the library's fused
attention under autograd (this package has no attention backward kernel yet), which costs one extra library forward.
For that reason the kernel is used for inference by default and for training only with ``KERAS_B200_FLASH_ATTENTION=1``;
otherwise the attention layers keep calling the library path (keras/src/backend/torch/nn.py:1124-1175).
"""

import ctypes
import os

import torch

from keras_b200.kernels import ops as kops

_ERR = {}


def _err_flag(device):
    t = _ERR.get(device.index)
    if t is None:
        t = _ERR[device.index] = torch.zeros(1, dtype=torch.int32, device=device)
    return t


def check_errors():
    for t in _ERR.values():
        code = int(t.item())
        if code != 0:
            t.zero_()
            raise RuntimeError(f"flash-attention kernel reported a pipeline time-out (code {code}).")


def _ok(t):
    return (t.is_cuda and t.dtype == torch.bfloat16 and t.ndim == 4 and t.stride(3) == 1 and t.data_ptr() % 16 == 0
            and all(s % 8 == 0 for s in t.stride()[:3]))


_V, _I, _L = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
_ARGUMENTS = [_V] * 5 + [_I] * 6 + [_L] * 12 + [ctypes.c_float, _I, _V] + [_L] * 3 + [_V, _L, _V, _V]
_LAUNCH = []


def _launcher():
    """The C entry with its argument types, so that a launch passes plain numbers: an object made for each of its 34
    (and row sums that nobody reads) cost 6 us a call, 24.5 -> 18.5."""
    if not _LAUNCH:
        fn = kops._lib().kb200_flash_attention_fwd
        fn.argtypes, fn.restype = _ARGUMENTS, ctypes.c_int
        _LAUNCH.append(fn)
    return _LAUNCH[0]


def forward(q, k, v, scale, is_causal, mask=None, row_mask=None, want_lse=True):
    """Raw kernel launch: returns ``(out [B, Tq, H, D] bf16, lse [B, H, Tq] fp32 or None)``.  ``mask``: bool ``[B, H, Tq, Tk]``, unit stride
    over the keys, any (also zero) strides over the rest; ``row_mask`` (with ``mask``): bool ``[B, Tq]``, unit stride over the rows."""
    B, Tq, H, D = q.shape
    Tk, Hkv = k.shape[1], k.shape[2]
    out = torch.empty((B, Tq, H, D), dtype=torch.bfloat16, device=q.device)
    lse = torch.empty((B, H, Tq), dtype=torch.float32, device=q.device) if want_lse else None
    (qb, qt, qh, _), (kb, kt, kh, _), (vb, vt, vh, _) = q.stride(), k.stride(), v.stride()
    # a dimension of one element may carry any stride: rows that are all the same are read once
    ms = (0, 0, 0) if mask is None else tuple(0 if n == 1 else s for n, s in zip(mask.shape[:3], mask.stride()))
    code = _launcher()(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr() if want_lse else None, B, Tq, Tk, H, Hkv, D, qt, qh, qb, kt, kh, kb,
                       vt, vh, vb, H * D, D, Tq * H * D, scale, 1 if is_causal else 0, mask.data_ptr() if mask is not None else None, ms[0], ms[1], ms[2],
                       row_mask.data_ptr() if row_mask is not None else None, row_mask.stride(0) if row_mask is not None else 0,
                       _err_flag(q.device).data_ptr(), kops._stream())
    kops._check(code, "flash_attention_fwd")
    return out, lse


class FlashAttentionFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, scale, is_causal):
        out, _ = forward(q, k, v, scale, is_causal, want_lse=False)
        ctx.save_for_backward(q, k, v)
        ctx.scale, ctx.is_causal = scale, is_causal
        return out

    @staticmethod
    def backward(ctx, grad_out):
        q, k, v = ctx.saved_tensors
        with torch.enable_grad():
            qq, kk, vv = (t.detach().requires_grad_(True) for t in (q, k, v))
            ref = torch.nn.functional.scaled_dot_product_attention(qq.transpose(1, 2), kk.transpose(1, 2), vv.transpose(1, 2), is_causal=ctx.is_causal,
                                                                   scale=ctx.scale, enable_gqa=qq.shape[2] != kk.shape[2])
            dq, dk, dv = torch.autograd.grad(ref, (qq, kk, vv), grad_out.transpose(1, 2))
        return dq, dk, dv, None, None


def _kernel_mask(mask, q, k, is_causal):
    """``mask`` (anything that broadcasts against ``[B, H, Tq, Tk]``) as the kernel reads it, the causal one included."""
    if mask.device != q.device or mask.ndim > 4 or mask.ndim == 0:
        return None
    mask = mask if mask.dtype == torch.bool else mask != 0
    if is_causal:
        mask = mask & torch.ones((q.shape[1], k.shape[1]), dtype=torch.bool, device=q.device).tril()
    try:
        if mask.shape[-1] != k.shape[1] or (mask.shape[-1] > 1 and mask.stride(-1) != 1):
            mask = mask.expand(tuple(mask.shape[:-1]) + (k.shape[1],)).contiguous()
        return mask.expand(q.shape[0], q.shape[2], q.shape[1], k.shape[1])
    except RuntimeError:
        return None


def flash_attention(q, k, v, mask, scale, is_causal, row_mask=None):
    """Attention on this package's kernel, or ``None`` when the call does not fit it (other head sizes, unaligned layouts, a scale
    that is not positive) or the kernel is not selected for training.

    ``row_mask`` (with ``mask``, not causal): bool ``[B, Tq]``; a row at zero has every key masked.  A padding mask as one byte a row
    and one a key, instead of their product over ``[B, Tq, Tk]``: 32 x 384 x 12 heads of 64 104 -> 50.5 us (unmasked 45.4)."""
    if row_mask is not None and (mask is None or is_causal or row_mask.dtype != torch.bool or row_mask.device != q.device
                                 or tuple(row_mask.shape) != tuple(q.shape[:2]) or row_mask.stride(1) != 1):
        return None
    if not (_ok(q) and _ok(k) and _ok(v)):
        return None
    # the kernel takes every size but the query's heads and rows from the query and the keys: what the library would broadcast is left to it
    D = q.shape[-1]
    if (D not in (64, 128) or k.shape != v.shape or k.shape[0] != q.shape[0] or k.shape[-1] != D or not q.device == k.device == v.device
            or 0 in q.shape or 0 in k.shape or q.shape[2] % k.shape[2]):
        return None
    needs_grad = torch.is_grad_enabled() and (q.requires_grad or k.requires_grad or v.requires_grad)
    mode = os.environ.get("KERAS_B200_FLASH_ATTENTION", "inference")
    if mode == "0" or (needs_grad and (mode != "1" or mask is not None)):
        return None
    if scale is None:
        scale = D ** -0.5
    if not scale > 0:
        return None
    if needs_grad:
        return FlashAttentionFn.apply(q, k, v, float(scale), bool(is_causal))
    if mask is not None:
        mask = _kernel_mask(mask, q, k, is_causal)
        if mask is None:
            return None
        is_causal = False
    return forward(q, k, v, float(scale), bool(is_causal), mask, row_mask, want_lse=False)[0]
