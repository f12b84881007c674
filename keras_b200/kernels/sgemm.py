"""Front-end of the float32 products of few rows (``csrc/sgemm.cu``): dense layers under the float32 policy.

A product, its bias and its rectifier are one launch; backward the rectifier's derivative and the bias gradient are one, and the weight
gradient is added where it is kept.  Larger layers, and any where the caller allows TF32 or is inside ``torch.autocast``, stay with the library.
"""

import ctypes

import torch

from keras_b200.kernels import ops as kops
from keras_b200.kernels import shadow

_i, _ll = ctypes.c_int, ctypes.c_longlong


def product(a, b, a_rows, b_rows, M, N, K, bias=None, relu=False, into=None):
    """``act(op(a) op(b) + bias)`` of 2-D float32 tensors with unit column strides, or ``into`` with the product added to it."""
    out = torch.empty((M, N), dtype=torch.float32, device=a.device) if into is None else into
    p = kops._p
    kops._check(kops._lib().kb200_sgemm(p(a), p(b), p(out), p(bias), _i(M), _i(N), _i(K), _ll(a.stride(0)), _ll(b.stride(0)), _ll(out.stride(0)), _i(1 if a_rows else 0),
                                        _i(1 if b_rows else 0), _i(1 if relu else 0), _i(0 if into is None else 1), kops._stream()), "sgemm")
    return out


def weight_gradient(a, b, target=None, bias_target=None, sums=False):
    """``(a^T b, column sums of b or None)`` of ``a [K, M]`` and ``b [K, N]``, float32 with unit column strides.  What could be added to
    its target's kept gradient comes back as ``None``."""
    (K, M), N = a.shape, b.shape[1]
    lib, p = kops._lib(), kops._p
    empty = lambda *shape: torch.empty(shape, dtype=torch.float32, device=b.device)  # noqa: E731
    slot = shadow.grad_slot(target, (M, N))
    db_slot = shadow.grad_slot(bias_target, (N,)) if sums else None
    c = empty(M, N) if slot is None else slot
    db = (empty(N) if db_slot is None else db_slot) if sums else None
    part = empty(lib.kb200_sgemm_wgrad_slices(_i(M), _i(N), _i(K)) * (M + 1) * ((N + 3) // 4 * 4))
    kops._check(lib.kb200_sgemm_wgrad(p(a), p(b), p(part), p(c), p(db), _i(M), _i(N), _i(K), _ll(a.stride(0)), _ll(b.stride(0)), _i(0 if slot is None else 1),
                                      _i(0 if db_slot is None else 1), kops._stream()), "sgemm_wgrad")
    return c if slot is None else None, db if db_slot is None else None


def _tf32():
    """Whether the caller lets the library round the operands of float32 products.  Asked by the newer of the two settings, which knows of both: once
    it is used, reading ``allow_tf32`` raises."""
    return torch.backends.cuda.matmul.fp32_precision not in ("none", "ieee")


def takes_weight_gradient(K, M, N, sums):
    """Whether ``weight_gradient`` is the quicker one, against the library's product and, with ``sums``, its column sums (us):

    with sums     6400 rows, 256 x 1024 118 -> 77; 128 rows, 256 x 1024 9.1 -> 7.6; beyond, 2000 rows, 512 x 2048 92 -> 107
    without       6400 rows, 32 x 1024 51 -> 17; few rows, 512 of 256 x 1024 11.3 -> 12.9; one column, 102400 of 1 x 400 45 -> 95
    many rows     102400 of 256 x 1024 with sums 1164 -> 1086, without 1066 -> 1086, and 1168 -> 1277 where 250 columns are copied singly"""
    if not 0 < M <= 256 or N <= 0 or K <= 0 or _tf32():
        return False
    if K > 32768 and M > 128 and (M % 4 or not sums):
        return False
    return sums or (K >= 1024 and M >= 8)


class DenseFn(torch.autograd.Function):
    """``relu?(x @ w + bias)``; ``w_target`` / ``bias_target``: the parameters themselves where their gradients may be added in place."""

    @staticmethod
    def forward(ctx, x, w, bias, w_target, bias_target, relu):
        M, K = x.shape
        N = w.shape[1]
        out = product(x, w, True, False, M, N, K, bias=bias, relu=relu)
        ctx.save_for_backward(x, w, bias, out if relu else None)
        ctx.targets, ctx.relu = (w_target, bias_target), relu
        return out

    @staticmethod
    def backward(ctx, dy):
        x, w, bias, out = ctx.saved_tensors
        need = ctx.needs_input_grad
        if torch.is_grad_enabled():  # a gradient of this gradient is wanted: differentiate the same layer from library operations
            operands = [t for t, n in zip((x, w, bias), need) if n]
            y = torch.matmul(x, w) if bias is None else torch.matmul(x, w) + bias
            grads = iter(torch.autograd.grad(torch.relu(y) if ctx.relu else y, operands, dy, create_graph=True))
            return tuple(next(grads) if n else None for n in need[:3]) + (None, None, None)
        M, K = x.shape
        N = w.shape[1]
        dy = dy.contiguous()
        p = kops._p
        db, slot = None, None
        if bias is not None and need[2]:
            slot = shadow.grad_slot(ctx.targets[1], (N,))
            db = slot.view(N) if slot is not None else torch.empty(N, dtype=torch.float32, device=dy.device)
        dz = torch.empty_like(dy) if ctx.relu else dy
        if ctx.relu or db is not None:
            kops._check(kops._lib().kb200_relu_bwd(p(dy), p(out), p(dz), p(db), _i(M), _i(N), _i(0 if slot is None else 1), kops._stream()), "relu_bwd")
        dx = product(dz, w, True, True, M, K, N) if need[0] else None
        dw = None
        if need[1]:
            g = shadow.grad_slot(ctx.targets[0], (K, N))
            made = product(x, dz, False, False, K, N, M, into=g.view(K, N) if g is not None else None)
            dw = made if g is None else None
        return dx, dw, db if slot is None else None, None, None, None


def _matrix(t):
    return type(t) in (torch.Tensor, torch.nn.Parameter) and t.is_cuda and t.dtype == torch.float32 and t.ndim == 2 and t.is_contiguous()


def dense(x, kernel, bias, activation_name):
    """``(output, activation_applied)`` or ``None``; ``kernel`` and ``bias`` are the layer's variables."""
    from keras_b200.core.variables import Variable

    # the type before any size: a traced batch has none yet
    if type(x) not in (torch.Tensor, torch.nn.Parameter) or type(kernel) is not Variable or kernel._shard_slices is not None or not (bias is None or type(bias) is Variable):
        return None
    w, b = kernel.value, None if bias is None else bias.value
    lead = x.shape[:-1]
    M = x.numel() // x.shape[-1] if x.shape[-1] else 0
    # Few rows and little work: the tiles are few and the split of K is what counts; beyond, the library's larger tiles are as quick or quicker.
    if not _matrix(w) or w.device != x.device or not 0 < M <= 256 or w.shape[0] != x.shape[-1] or w.shape[0] < 16 or w.shape[1] == 0 or M * w.numel() > 1 << 27:
        return None
    if _tf32() or torch.is_autocast_enabled("cuda") or (b is not None and (b.dtype != torch.float32 or b.device != x.device or not b.is_contiguous())):
        return None
    x2 = x.reshape(M, w.shape[0])
    if not _matrix(x2):
        return None
    relu = activation_name == "relu"
    done = relu or activation_name in (None, "linear")
    if torch.is_grad_enabled() and (x2.requires_grad or w.requires_grad or (b is not None and b.requires_grad)):
        targets = [v._value if v is not None and t is v._value and t.requires_grad else None for v, t in ((kernel, w), (bias, b))]
        out = DenseFn.apply(x2, w, b, targets[0], targets[1], relu)
    else:
        out = product(x2, w, True, False, M, w.shape[1], w.shape[0], bias=b, relu=relu)
    return out.reshape(tuple(lead) + (w.shape[1],)), done
