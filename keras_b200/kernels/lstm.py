"""Front-end of the whole-sequence LSTM kernels (``csrc/lstm.cu``).

``run`` takes the projected inputs of all time steps and returns the outputs, the last state and the last cell state of a stock
LSTM layer (keras/src/layers/rnn/lstm.py:240-300) from one launch; its backward pass is one launch and the weight gradients.
"""

import ctypes

import torch

from keras_b200.kernels import ops as kops
from keras_b200.kernels import sgemm
from keras_b200.kernels.gemm import _err_flag

_i = ctypes.c_int


def _plain(t):
    return type(t) in (torch.Tensor, torch.nn.Parameter) and t.is_cuda and t.dtype == torch.float32


def _groups(batch, units):
    return kops._lib().kb200_lstm_groups(_i(batch), _i(units))


def takes(sequences, initial_state, cell):
    """float32 tensors on one device, a batch and a width that the launch holds; no ``torch.autocast``, whose products are 16-bit."""
    if torch.is_autocast_enabled("cuda") or not _plain(sequences) or sequences.ndim != 3 or sequences.shape[0] == 0 or sequences.shape[1] == 0 or len(initial_state) != 2:
        return False
    weights = [cell.kernel, cell.recurrent_kernel] + ([cell.bias] if cell.bias is not None else [])
    if any(getattr(w, "_shard_slices", None) is not None for w in weights):
        return False
    tensors = [w.value if hasattr(w, "value") else w for w in weights] + list(initial_state)
    if not all(isinstance(t, torch.Tensor) and _plain(t) and t.device == sequences.device for t in tensors):
        return False
    shape = (sequences.shape[0], cell.units)
    return all(tuple(s.shape) == shape for s in initial_state) and _groups(*shape) > 0


def _composed(xz, bias, h, c, R, reverse):
    """The same layer from torch operations: ``(outputs in processing order, last h, last c)``."""
    u = R.shape[0]
    outs = []
    steps = range(xz.shape[1] - 1, -1, -1) if reverse else range(xz.shape[1])
    for t in steps:
        z = xz[:, t] + torch.matmul(h, R) if bias is None else xz[:, t] + bias + torch.matmul(h, R)
        i, f, g, o = z[:, :u].sigmoid(), z[:, u:2 * u].sigmoid(), z[:, 2 * u:3 * u].tanh(), z[:, 3 * u:].sigmoid()
        c = f * c + i * g
        h = o * c.tanh()
        outs.append(h)
    return torch.stack(outs, dim=1), h, c


def _launch(backward, xz, bias, h0, c0, R, hprev, out, hT, cT, gates, cs, dout, dhT, dcT, dz, dh0, dc0, reverse):
    B, T, U = xz.shape[0], xz.shape[1], R.shape[0]
    counters = None if kops._lib().kb200_lstm_clustered(_i(B), _i(U), _i(backward)) else torch.zeros(_groups(B, U), dtype=torch.int32, device=xz.device)
    p = kops._p
    code = kops._lib().kb200_lstm(_i(backward), p(xz), p(bias), p(h0), p(c0), p(R), p(hprev), p(out), p(hT), p(cT), p(gates), p(cs), p(dout), p(dhT), p(dcT),
                                  p(dz), p(dh0), p(dc0), p(counters), p(_err_flag(xz.device)), _i(B), _i(T), _i(U), _i(1 if reverse else 0), kops._stream())
    kops._check(code, "lstm")


def _aligned(t):
    """Contiguous and 16-byte aligned: the kernels read rows of the state and of its gradient as vectors."""
    t = t.detach().contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


class Project(torch.autograd.Function):
    """``x @ W`` of every time step, its weight gradient by the kernel for products over many rows."""

    @staticmethod
    def forward(ctx, x, W, target):
        ctx.save_for_backward(x, W)
        ctx.target = target
        return torch.matmul(x, W)

    @staticmethod
    def backward(ctx, dxz):
        x, W = ctx.saved_tensors
        need = ctx.needs_input_grad
        if torch.is_grad_enabled():  # a gradient of this gradient is wanted: differentiate the library's product
            grads = iter(torch.autograd.grad(torch.matmul(x, W), [t for t, n in zip((x, W), need) if n], dxz, create_graph=True))
            return tuple(next(grads) if n else None for n in need[:2]) + (None,)
        rows, dz = x.reshape(-1, x.shape[-1]), dxz.reshape(-1, dxz.shape[-1]).contiguous()
        dW = None
        if need[1]:
            if sgemm.takes_weight_gradient(rows.shape[0], rows.shape[1], dz.shape[1], False):
                dW, _ = sgemm.weight_gradient(rows.contiguous(), dz, ctx.target)
            else:
                dW = torch.matmul(rows.t(), dz)
        return torch.matmul(dxz, W.t()) if need[0] else None, dW, None


def _target(variable, tensor):
    """The parameter itself where a kernel may add its gradient in place, else ``None``."""
    return tensor if tensor is not None and getattr(variable, "_value", None) is tensor and tensor.requires_grad else None


def project(sequences, kernel):
    """The projected inputs of all time steps, for operands that ``takes`` has let through."""
    W = kernel.value if hasattr(kernel, "value") else kernel
    if torch.is_grad_enabled() and W.requires_grad and W.ndim == 2 and W.shape[0] == sequences.shape[-1]:
        return Project.apply(sequences, W, _target(kernel, W))
    return torch.matmul(sequences, W)


class LstmSequence(torch.autograd.Function):
    @staticmethod
    def forward(ctx, xz, bias, h0, c0, R, reverse, want_sequence, recording, bias_target=None, R_target=None):
        B, T = xz.shape[0], xz.shape[1]
        U = R.shape[0]
        x, h, c, r = _aligned(xz), _aligned(h0), _aligned(c0), _aligned(R)
        b = bias.detach().contiguous() if bias is not None else None
        # needs_input_grad follows requires_grad whether gradients are recorded or not: trainable weights have it in inference too
        grad = recording and any(ctx.needs_input_grad)
        empty = lambda *shape: torch.empty(shape, dtype=torch.float32, device=xz.device)  # noqa: E731
        hprev, hT, cT = empty(B, T, U), empty(B, U), empty(B, U)
        out = empty(B, T, U) if want_sequence else None
        gates, cs = (empty(T, B, 4 * U), empty(T, B, U)) if grad else (None, None)
        _launch(0, x, b, h, c, r, hprev, out, hT, cT, gates, cs, None, None, None, None, None, None, reverse)
        ctx.save_for_backward(xz, bias, h0, c0, R, hprev, gates, cs)
        ctx.reverse, ctx.targets = reverse, (bias_target, R_target)
        ctx.set_materialize_grads(False)
        return out, hT, cT

    @staticmethod
    def backward(ctx, dout, dhT, dcT):
        xz, bias, h0, c0, R, hprev, gates, cs = ctx.saved_tensors
        if dout is None and dhT is None and dcT is None:
            return (None,) * 10
        if torch.is_grad_enabled():  # a gradient of this gradient is wanted: differentiate the composed operations
            inputs = [xz, bias, h0, c0, R]
            wanted = [t for t, need in zip(inputs, ctx.needs_input_grad) if need]
            results = _composed(xz, bias, h0, c0, R, ctx.reverse)
            pairs = [(r, g) for r, g in zip(results, (dout, dhT, dcT)) if g is not None]
            grads = iter(torch.autograd.grad([r for r, _ in pairs], wanted, [g for _, g in pairs], create_graph=True, allow_unused=True))
            return tuple(next(grads) if need else None for need in ctx.needs_input_grad[:5]) + (None,) * 5
        B, T, U = hprev.shape
        need = ctx.needs_input_grad
        dout, dhT, dcT = (g.contiguous() if g is not None else None for g in (dout, dhT, dcT))
        dz = torch.empty_like(xz, memory_format=torch.contiguous_format)
        dc0 = torch.empty((B, U), dtype=torch.float32, device=xz.device)
        dh0 = torch.empty_like(dc0) if need[2] else None
        _launch(1, xz, None, None, c0.detach().contiguous(), R.detach().contiguous(), None, None, None, None, gates, cs, dout, dhT, dcT, dz, dh0, dc0,
                ctx.reverse)
        flat = dz.view(B * T, 4 * U)
        if need[4] and sgemm.takes_weight_gradient(B * T, U, 4 * U, need[1]):
            dR, db = sgemm.weight_gradient(hprev.view(B * T, U), flat, ctx.targets[1], ctx.targets[0], sums=need[1])
        else:
            dR = torch.matmul(hprev.view(B * T, U).t(), flat) if need[4] else None
            db = flat.sum(0) if need[1] else None
        return (dz if need[0] else None, db, dh0, dc0 if need[3] else None, dR) + (None,) * 5


def run(xz, bias, h0, c0, R, reverse, want_sequence, bias_target=None, R_target=None):
    """``(outputs [B, T, U] in processing order or None, last h, last c)``; targets as ``_target`` finds them."""
    return LstmSequence.apply(xz, bias, h0, c0, R, bool(reverse), bool(want_sequence), torch.is_grad_enabled(), bias_target, R_target)


def layer(sequences, cell, h0, c0, reverse, want_sequence):
    """``run`` on the inputs of a stock cell that ``takes`` has let through."""
    (bias, R), xz = [(v.value if hasattr(v, "value") else v) for v in (cell.bias, cell.recurrent_kernel)], project(sequences, cell.kernel)
    return run(xz, bias, h0, c0, R, reverse, want_sequence, _target(cell.bias, bias), _target(cell.recurrent_kernel, R))
