"""Front-end of the depthwise convolution kernels (``csrc/depthwise.cu``).

``depthwise`` returns ``None`` when a call does not meet the kernels' contract (bf16 on CUDA, channels last, one output per input
channel, square filters of 3, 5 or 7 taps with stride 1 or 2 and no dilation, channels a multiple of 8); the caller then uses
the grouped library convolution (keras/src/backend/torch/nn.py:717-760).
"""

import torch

from keras_b200.kernels import ops as kops
from keras_b200.kernels import shadow
from keras_b200.kernels.conv import _target_param


def _launch(mode, x, w, y, dy, dw, g, accumulate=True):
    N, H, W, C, OH, OW, K, S, pt, pl = g
    i, p = kops._i, kops._p
    lib, partial = kops._lib(), None
    if mode == 2:
        partial = torch.empty((lib.kb200_depthwise_slabs(i(N), i(OH), i(OW), i(C), i(K)), K * K * C), dtype=torch.float32, device=x.device)
    code = lib.kb200_depthwise(i(mode), p(x), p(w), p(y), p(dy), p(dw), p(partial), i(1 if accumulate else 0), i(N), i(H), i(W), i(C), i(OH), i(OW), i(K),
                               i(S), i(pt), i(pl), kops._stream())
    kops._check(code, "depthwise")


def _aligned(t):
    t = t.detach().contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _composed(x, w, g):
    """The same convolution from library operations (used to differentiate a gradient)."""
    N, H, W, C, OH, OW, K, S, pt, pl = g
    pad = (pl, max((OW - 1) * S + K - W - pl, 0), pt, max((OH - 1) * S + K - H - pt, 0))
    xc = torch.nn.functional.pad(x.permute(0, 3, 1, 2), pad)
    return torch.nn.functional.conv2d(xc, w.permute(2, 3, 0, 1), stride=S, groups=C)[:, :, :OH, :OW].permute(0, 2, 3, 1)


class DepthwiseFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, g, grad_target):
        N, H, W, C, OH, OW, K, S, pt, pl = g
        y = torch.empty((N, OH, OW, C), dtype=torch.bfloat16, device=x.device)
        _launch(0, _aligned(x), _aligned(w), y, None, None, g)
        ctx.save_for_backward(x, w)
        ctx.g, ctx.grad_target = g, grad_target
        return y

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        g = ctx.g
        N, H, W, C, OH, OW, K, S, pt, pl = g
        if torch.is_grad_enabled():  # a gradient of this gradient is wanted
            wanted = [t for t, need in zip((x, w), ctx.needs_input_grad) if need]
            grads = iter(torch.autograd.grad(_composed(x, w, g), wanted, dy, create_graph=True))
            return tuple(next(grads) if need else None for need in ctx.needs_input_grad[:2]) + (None, None)
        dy = _aligned(dy if dy.dtype == torch.bfloat16 else dy.to(torch.bfloat16))
        dx = dw = None
        if ctx.needs_input_grad[0]:
            dx = torch.empty((N, H, W, C), dtype=torch.bfloat16, device=dy.device)
            _launch(1, dy, _aligned(w), dx, None, None, g)
        if ctx.needs_input_grad[1]:
            slot = shadow.grad_slot(ctx.grad_target, w.shape)
            buf = slot if slot is not None else torch.empty(w.shape, dtype=torch.float32, device=dy.device)
            _launch(2, _aligned(x), None, None, dy, buf, g, accumulate=slot is not None)
            dw = buf.to(w.dtype) if slot is None else None  # already inside the parameter's gradient
        return dx, dw, None, None


def depthwise(x, kernel, strides, padding, data_format, dilation, variable=None):
    """``variable``: the ``Variable`` that ``kernel`` was read from; a gradient that lives in persistent fp32 storage is added to there."""
    if (data_format != "channels_last" or type(x) is not torch.Tensor or not isinstance(kernel, torch.Tensor) or x.ndim != 4 or kernel.ndim != 4
            or x.dtype != torch.bfloat16 or kernel.dtype != torch.bfloat16 or not isinstance(padding, str)):
        return None
    N, H, W, C = x.shape
    K, K2, cin, mult = kernel.shape
    sh, sw = strides
    if K != K2 or K not in (3, 5, 7) or cin != C or mult != 1 or C % 8 or sh != sw or sh not in (1, 2) or tuple(dilation) != (1, 1):
        return None
    mode = padding.lower()
    if mode == "same":
        OH, OW = -(-H // sh), -(-W // sh)
        pt, pl = (max((o - 1) * sh + K - n, 0) // 2 for o, n in ((OH, H), (OW, W)))
    elif mode == "valid":
        OH, OW, pt, pl = (H - K) // sh + 1, (W - K) // sh + 1, 0, 0
    else:
        return None
    if N == 0 or OH <= 0 or OW <= 0 or N * H * W >= 1 << 30 or N * OH * OW >= 1 << 30:
        return None
    if sh == 1 and K == 3 and not (torch.is_grad_enabled() and (x.requires_grad or kernel.requires_grad)):
        # the forward pass alone: without a stride nothing is padded or re-laid, and the library's 3x3 kernel takes 0.86 of this one's
        # time (28x28x192 31 us against 35; 5x5 66 / 61, 7x7 at 56x56x96 115 / 109); with gradients these kernels take 0.6 of its
        return None
    target = _target_param(variable, kernel) if variable is not None and kernel.is_contiguous() else None
    return DepthwiseFn.apply(x, kernel, (N, H, W, C, OH, OW, K, sh, pt, pl), target)
