"""Front-end of the tcgen05 bf16 GEMM (``csrc/gemm_sm100.cu``): autograd function and dispatch rules.

``matmul`` / ``dense`` return ``None`` when an operand does not meet the kernel's contract (bf16 on
CUDA, 16-byte aligned, row pitches multiples of 8 elements); callers then use ``torch.matmul``.
The three products of a dense layer map to operand-major flags of the same kernel:

    forward   C  = X  · W        A K-major,  B MN-major
    dgrad     dX = dY · Wᵀ       A K-major,  B K-major
    wgrad     dW = Xᵀ · dY       A MN-major, B MN-major
"""

import ctypes
import os

import torch

from keras_b200.kernels import ops as kops
from keras_b200.kernels import shadow

_ACT = {None: 0, "linear": 0, "relu": 1, "gelu_tanh": 2, "silu": 3, "swish": 3, "gelu_erf": 4}
_ERR = {}
_MIN_WORK = int(os.environ.get("KERAS_B200_GEMM_MIN_FLOPS", str(1 << 22)))
# measured on GPT-2 (launch-bound step): 2 % slower than the bf16 gradient + one add, so off unless asked for
_WGRAD_IN_PLACE = os.environ.get("KERAS_B200_WGRAD_IN_PLACE", "1") == "1"


def _err_flag(device):
    key = (device.type, device.index)
    t = _ERR.get(key)
    if t is None:
        t = torch.zeros(1, dtype=torch.int32, device=device)
        _ERR[key] = t
    return t


def check_errors():
    """Raise if any GEMM launch gave up on a bounded wait (reads the device flag: synchronises)."""
    for t in _ERR.values():
        code = int(t.item())
        if code != 0:
            t.zero_()
            raise RuntimeError(f"tcgen05 GEMM reported a pipeline time-out (code {code}).")


def _ok_2d(t, any_width=False):
    if any_width and t.is_cuda and t.dtype == torch.bfloat16 and t.ndim == 2 and t.is_contiguous() and t.data_ptr() % 16 == 0:
        return True  # a weight whose width is padded to a multiple of 8 before the launch
    return t.is_cuda and t.dtype == torch.bfloat16 and t.ndim == 2 and t.stride(1) == 1 and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0 and t.stride(0) >= t.shape[1]


_SM_COUNT = {}


def _sm_count(device):
    n = _SM_COUNT.get(device.index)
    if n is None:
        n = _SM_COUNT[device.index] = torch.cuda.get_device_properties(device).multi_processor_count
    return n


def split_k_for(M, N, K, device):
    """K slices for an accumulated product (weight gradients: small M x N, K = tokens), which add their tiles as they come; so only where there
    is much to gain, and the other products repeat bit for bit.  Those with the least waves x (K blocks + 10), the ten for a unit's start and
    for adding its tile.  Against the time of 1 to 20 slices at eleven sizes it finds the best within 4 %: [768, 2304, 16384] 55.2 -> 46.8 us in five
    slices (two, which fill a wave to three quarters, before), [512, 512, 2664] 10.1 -> 8.8.  Few tiles over very many rows take all SMs: cold,
    [512, 64, 200704] 58 us in 37 slices and 86 in 16, [32, 24, 100352] 17 in 143 and 44."""
    sms = _sm_count(device)
    one, pair, blocks = -(-M // 128) * -(-N // 256), -(-M // 256) * -(-N // 256), -(-K // 64)
    if one * 2 > sms or K < 2048:
        return 1
    best, slices = None, 1
    for s in range(1, min(max(16, sms // one), blocks // 3) + 1):
        per = -(-blocks // s)
        if per * (s - 1) >= blocks:
            continue  # fewer slices hold as much
        # the kernels' own rule (gemm_variant): pairs from nine tenths of a wave of them
        paired = M > 128 and N > 128 and pair * s * 10 >= sms // 2 * 9 and -(-pair * s // (sms // 2)) <= -(-one * s // sms)
        waves = -(-pair * s // (sms // 2)) if paired else -(-one * s // sms)
        cost = waves * (per + 10)
        if best is None or cost < best:
            best, slices = cost, s
    return slices


def input_gradient_slices(M, K, N, device):
    """K slices for dX[M, K] = dY[M, N] W^T, whose result is bf16: a few tiles that each walk a vocabulary are worth float32 results of their own and
    a pass that adds them, in order ([2664, 512, 8009] 37.8 -> 28.9 us, [300, 768, 50257] 492 -> 56; [4096, 512, 8009] 38.3 and 39.8)."""
    tiles = -(-M // 128) * -(-K // 256)
    slices = min(_sm_count(device) // tiles, N // 512, 16)
    return slices if N >= 4096 and slices >= 3 else 1


def input_gradient(dy, w, M, K, N):
    """``dy @ w^T``, the sum over ``N`` columns, in bf16; the same bits every time."""
    slices = input_gradient_slices(M, K, N, dy.device)
    if slices == 1 or K % 8:
        return gemm(dy, w, 0, 0, M, K, N)
    lib = kops._lib()
    lib.kb200_gemm_slices_floats.restype = ctypes.c_longlong
    part = torch.empty(lib.kb200_gemm_slices_floats(kops._i(M), kops._i(K), kops._i(slices)), dtype=torch.float32, device=dy.device)
    out = torch.empty((M, K), dtype=torch.bfloat16, device=dy.device)
    code = lib.kb200_gemm_bf16_slices(kops._p(dy), kops._p(w), kops._p(out), kops._p(part), kops._i(M), kops._i(K), kops._i(N), kops._ll(dy.stride(0)), kops._ll(w.stride(0)),
                                      kops._i(0), kops._i(0), kops._i(slices), kops._p(_err_flag(dy.device)), kops._stream())
    kops._check(code, "gemm_bf16_slices")
    return out


def gemm(a, b, a_mn, b_mn, M, N, K, bias=None, act=0, out_dtype=torch.bfloat16, split_k=1, accumulate_into=None):
    """Raw launch. ``a``/``b`` are 2-D bf16 tensors in the storage layout named by the major flags.

    ``split_k > 1`` accumulates K slices into a zeroed fp32 buffer (TMA reduce stores) and casts to ``out_dtype``.
    ``bias``: fp32 or bf16.
    ``accumulate_into``: fp32 [M, N] tensor that the product is added to in place (returned)."""
    lib = kops._lib()
    err = _err_flag(a.device)
    if accumulate_into is not None:
        acc = accumulate_into
        code = lib.kb200_gemm_bf16_run(kops._p(a), kops._p(b), kops._p(acc), None, kops._i(M), kops._i(N), kops._i(K), kops._ll(a.stride(0)),
                                       kops._ll(b.stride(0)), kops._ll(acc.stride(0)), kops._i(a_mn), kops._i(b_mn), kops._i(0), kops._i(1),
                                       kops._i(0), kops._i(-max(1, split_k)), kops._i(0), kops._p(err), kops._stream())
        kops._check(code, "gemm_bf16")
        return acc
    if split_k > 1 and bias is None and act == 0:
        acc = torch.zeros((M, N), dtype=torch.float32, device=a.device)
        code = lib.kb200_gemm_bf16_run(kops._p(a), kops._p(b), kops._p(acc), None, kops._i(M), kops._i(N), kops._i(K), kops._ll(a.stride(0)),
                                       kops._ll(b.stride(0)), kops._ll(acc.stride(0)), kops._i(a_mn), kops._i(b_mn), kops._i(0), kops._i(1),
                                       kops._i(0), kops._i(split_k), kops._i(0), kops._p(err), kops._stream())
        kops._check(code, "gemm_bf16")
        return acc if out_dtype == torch.float32 else acc.to(out_dtype)
    out = torch.empty((M, N), dtype=out_dtype, device=a.device)
    code = lib.kb200_gemm_bf16_run(kops._p(a), kops._p(b), kops._p(out), kops._p(bias), kops._i(M), kops._i(N), kops._i(K),
                                   kops._ll(a.stride(0)), kops._ll(b.stride(0)), kops._ll(out.stride(0)), kops._i(a_mn), kops._i(b_mn), kops._i(act),
                                   kops._i(1 if out_dtype == torch.float32 else 0), kops._i(1 if bias is not None and bias.dtype == torch.bfloat16 else 0),
                                   kops._i(1), kops._i(0), kops._p(err), kops._stream())
    kops._check(code, "gemm_bf16")
    return out


_ACT_FN = {1: torch.relu, 3: torch.nn.functional.silu, 4: torch.nn.functional.gelu}


def _bias_operand(bias):
    """A bias as the epilogue reads it: fp32 or bf16, contiguous."""
    if bias is None:
        return None
    return (bias if bias.dtype in (torch.float32, torch.bfloat16) else bias.float()).detach().contiguous()


def padded_width(N):
    """Columns that a product of odd width is computed in: multiples of 8 as the copies need them, and of 64 beyond a thousand, where that is
    no tile and at most a sixteenth more.  Rows then start on 128-byte lines, and a tile's 128 bytes of a row are one line, not two.
    [16384, 768] by a vocabulary of 50257 in 50264 and 50304 columns: product 1118 and 1015 us, input gradient 1088 and 900."""
    return (N + 7) // 8 * 8 if N % 8 == 0 or N <= 1024 else (N + 63) // 64 * 64


class GemmFn(torch.autograd.Function):
    """out[M,N] = x[M,K] @ w[K,N] (+ bias), all three products on the tcgen05 kernel.

    A width ``N`` that is not a multiple of 8 (a 50257-word vocabulary) runs on a zero-padded copy of the weight:
    the padded output keeps its 16-byte row pitch and the caller sees its first ``N`` columns as a view."""

    @staticmethod
    def forward(ctx, x, w, bias, grad_target=None, bias_target=None, act=0):
        """``act``: code of the activation behind the product (relu, silu, gelu): its derivative and the bias gradient are one pass.
        (Its value as a second output of the epilogue gains 12 of 130 us at [16384, 3072, 768] and nothing at smaller products.)
        ``grad_target``: the fp32 parameter behind ``w`` (its bf16 shadow) when its ``.grad`` is persistent fp32 storage: the
        weight gradient is then accumulated there by the GEMM itself and no bf16 gradient tensor is produced."""
        M, K = x.shape
        N = w.shape[1]
        ctx.grad_target = grad_target
        ctx.bias_target = bias_target
        Np = padded_width(N)
        b = _bias_operand(bias)
        wide = w
        if Np != N:
            wide = kops.pad_columns(w, Np)
            if b is not None:
                b = torch.nn.functional.pad(b, (0, Np - N))
        out, pre = gemm(x, wide, 0, 1, M, Np, K, bias=b), None
        if act:
            pre, out = out, kops.gelu(out) if act == 4 else _ACT_FN[act](out)
        ctx.save_for_backward(x, w, bias, pre, wide if Np != N else None)
        ctx.act = act
        ctx.has_bias = bias is not None
        ctx.bias_dtype = bias.dtype if bias is not None else None
        ctx.n = N
        return out if Np == N else out[:, :N]

    @staticmethod
    def backward(ctx, dy):
        x, w, bias, pre, wide = ctx.saved_tensors
        if torch.is_grad_enabled():  # a gradient of this gradient is wanted: differentiate the same layer from library operations
            operands = [t for t, need in zip((x, w, bias), ctx.needs_input_grad) if need]
            out = torch.matmul(x, w) if bias is None else torch.matmul(x, w) + bias.to(x.dtype)
            grads = iter(torch.autograd.grad(_ACT_FN[ctx.act](out) if ctx.act else out, operands, dy, create_graph=True))
            return tuple(next(grads) if need else None for need in ctx.needs_input_grad[:3]) + (None,) * (len(ctx.needs_input_grad) - 3)
        w = w if wide is None else wide
        M, K = x.shape
        N, Np = ctx.n, w.shape[1]
        sums = bias_slot = None
        if ctx.act:
            dy = kops.aligned(dy)
            wanted = ctx.has_bias and ctx.needs_input_grad[2]
            bias_slot = shadow.grad_slot(ctx.bias_target, (N,)) if wanted else None
            dy, sums = kops.activation_backward(dy, pre, ctx.act, wanted, bias_slot.view(N) if bias_slot is not None else None)
        if Np != N:
            if (dy.dtype == torch.bfloat16 and dy.stride(1) == 1 and dy.stride(0) == Np and dy.data_ptr() % 16 == 0
                    and (dy.storage_offset() + M * Np) * dy.element_size() <= dy.untyped_storage().nbytes()):
                # The gradient is itself the leading columns of a wider buffer, often the padded logits' own.  What stands in the columns
                # behind may be somebody else's (a concatenation's other operand): it is neither written nor summed over.
                dy = dy.as_strided((M, Np), (Np, 1))
            else:
                wide_dy = torch.empty((M, Np), dtype=torch.bfloat16, device=dy.device)
                wide_dy[:, :N].copy_(dy)
                wide_dy[:, N:].zero_()
                dy = wide_dy
        elif not _ok_2d(dy):
            dy = kops.aligned(dy)
        dx = dw = db = None
        if ctx.needs_input_grad[0]:
            dx = input_gradient(dy, w, M, K, N)  # the sum ends at N; below, the columns behind it stay columns of their own
        if ctx.needs_input_grad[1]:
            split = split_k_for(K, Np, M, x.device)
            g = shadow.grad_slot(ctx.grad_target, (K, N)) if Np == N and N % 4 == 0 else None
            if g is not None:
                gemm(x, dy, 1, 1, K, N, M, split_k=split, accumulate_into=g.view(K, N))  # dw stays None: already accumulated
            else:
                dw = gemm(x, dy, 1, 1, K, Np, M, split_k=split)
                if Np != N:
                    dw = dw[:, :N]
        if sums is not None:
            db = sums.to(ctx.bias_dtype) if bias_slot is None else None
        elif ctx.has_bias and ctx.needs_input_grad[2]:
            g = shadow.grad_slot(ctx.bias_target, (N,)) if Np == N else None
            if g is not None:
                kops.column_sum(dy, accumulate_into=g.view(N))  # db stays None: already accumulated
            else:
                db = kops.column_sum(dy)[:N].to(ctx.bias_dtype)
        return (dx, dw, db, None, None, None)[: len(ctx.needs_input_grad)]


def group(products, M, a_mn, b_mn, sum_k, split_k=1, accumulate=False):
    """One launch for up to three products, each ``(a, b, c, bias)``: side by side (``c`` of their own, one ``a``), or summed into the first
    one's ``c``.  ``N`` and ``K`` are read from ``b`` as the major flag says.  ``accumulate``: added to what the float32 ``c`` hold."""
    lib = kops._lib()
    n = len(products)
    a0, _, c0, _ = products[0]
    pointers, sizes, pitches = (ctypes.c_void_p * (4 * n))(), (ctypes.c_int * (2 * n))(), (ctypes.c_longlong * (3 * n))()
    for i, (a, b, c, bias) in enumerate(products):
        c = c0 if sum_k else c
        pointers[4 * i:4 * i + 4] = [a.data_ptr(), b.data_ptr(), c.data_ptr(), bias.data_ptr() if bias is not None else None]
        sizes[2 * i:2 * i + 2] = [b.shape[1], b.shape[0]] if b_mn else [b.shape[0], b.shape[1]]
        pitches[3 * i:3 * i + 3] = [a.stride(0), b.stride(0), c.stride(0)]
    bias16 = any(p[3] is not None and p[3].dtype == torch.bfloat16 for p in products)
    code = lib.kb200_gemm_group(pointers, sizes, pitches, kops._i(n), kops._i(1 if sum_k else 0), kops._i(M), kops._i(a_mn), kops._i(b_mn),
                                kops._i(1 if c0.dtype == torch.float32 else 0), kops._i(1 if bias16 else 0), kops._i(-max(1, split_k) if accumulate else split_k),
                                kops._i(0), kops._p(_err_flag(a0.device)), kops._stream())
    kops._check(code, "gemm_group")


class ProjectionsFn(torch.autograd.Function):
    """``x @ w_i (+ bias_i)`` for the three projections of an attention layer: one launch forward, one for the gradient of ``x`` (a sum over
    the three in fp32, where three results in bf16 were added afterwards) and one for the weights' gradients."""

    @staticmethod
    def forward(ctx, x, targets, w0, w1, w2, *biases):
        ws = (w0, w1, w2)
        M = x.shape[0]
        outs = [torch.empty((M, w.shape[1]), dtype=torch.bfloat16, device=x.device) for w in ws]
        group([(x, w, o, b) for w, o, b in zip(ws, outs, [b.detach() for b in biases] or [None] * 3)], M, 0, 1, False)
        ctx.save_for_backward(x, *ws, *biases)
        ctx.targets = targets  # the parameters behind weights and biases, where their gradients may be added in place
        return tuple(outs)

    @staticmethod
    def backward(ctx, *dys):
        x, *rest = ctx.saved_tensors
        ws, biases = rest[:3], rest[3:]
        need = ctx.needs_input_grad
        if torch.is_grad_enabled():  # a gradient of this gradient is wanted: differentiate the same products from library operations
            operands = [t for t, n in zip((x, *ws, *biases), (need[0], *need[2:])) if n]
            outs = [torch.matmul(x, w) + (biases[i] if biases else 0) for i, w in enumerate(ws)]
            grads = iter(torch.autograd.grad(outs, operands, dys, create_graph=True))
            picked = [next(grads) if n else None for n in (need[0], *need[2:])]
            return (picked[0], None, *picked[1:])
        dys = [dy if _ok_2d(dy) else kops.aligned(dy) for dy in dys]
        M, K = x.shape
        dx = None
        if need[0]:
            dx = torch.empty((M, K), dtype=torch.bfloat16, device=x.device)
            group([(dy, w, dx, None) for dy, w in zip(dys, ws)], M, 0, 0, True)
        dws = [None] * 3
        if any(need[2:5]):
            slots = [shadow.grad_slot(t, w.shape) if n else None for t, w, n in zip(ctx.targets[:3], ws, need[2:5])]
            if all(s is not None for s in slots):
                split = split_k_for(K, sum(w.shape[1] for w in ws), M, x.device)
                group([(x, dy, s.view(w.shape), None) for dy, w, s in zip(dys, ws, slots)], K, 1, 1, False, split_k=split, accumulate=True)
            else:
                for i, (dy, w, s) in enumerate(zip(dys, ws, slots)):
                    if need[2 + i]:
                        into = s.view(w.shape) if s is not None else None
                        made = gemm(x, dy, 1, 1, K, w.shape[1], M, split_k=split_k_for(K, w.shape[1], M, x.device), accumulate_into=into)
                        dws[i] = made if s is None else None
        dbs = [None] * len(biases)
        for i, b in enumerate(biases):
            if need[5 + i]:
                s = shadow.grad_slot(ctx.targets[3 + i], b.shape)
                made = kops.column_sum(dys[i], accumulate_into=s.view(-1) if s is not None else None)
                dbs[i] = made.to(b.dtype) if s is None else None
        return (dx, None, *dws, *dbs)


def projections(x, kernels, biases, weights):
    """The three projections of ``x`` [..., K] by ``kernels`` (variables that read as ``weights``, [K, heads, size]) as [..., heads, size], or
    ``None`` where their products do not fit one launch."""
    K = x.shape[-1]
    x2 = x.reshape(-1, K)
    flat = [w.reshape(K, -1) for w in weights]
    if K % 64 or any(w.shape[1] % 64 or not _qualifies(x2, w) for w in flat):
        return None
    bs = [b.value.reshape(-1) for b in biases]
    if any(b.device != x.device or b.dtype != bs[0].dtype or b.dtype not in (torch.float32, torch.bfloat16) or not b.is_contiguous() for b in bs):
        return None
    targets = [_grad_target(k, w) for k, w in zip(kernels, weights)] + [_grad_target(v, b) for v, b in zip(biases, bs)]
    outs = ProjectionsFn.apply(x2, targets, *flat, *bs)
    return tuple(o.reshape(tuple(x.shape[:-1]) + tuple(w.shape[1:])) for o, w in zip(outs, weights))


def _qualifies(x2, w):
    if not (_ok_2d(x2) and _ok_2d(w, any_width=True)) or w.device != x2.device:
        return False
    M, K = x2.shape
    return takes(M, w.shape[1], K)


def takes(M, N, K):
    """Whether products of this size run here: the others are the library's."""
    # Rows may be any number: the copies clip them.  Up to a tile of them the library's small-batch kernels take half of this one's time
    # ([77, 3072, 768] 6.0 us against 13.2, [77, 768, 3072] 3.6 / 6.2, [77, 768, 50264] 12 / 20; 72 to 128 rows the same), and row counts that
    # are no multiple of 8 go to them; multiples of 8 do not, a line that time did not draw.  A width that is no multiple of 8 would send
    # the library to kernels of three generations ago ([77, 768, 50257] 100 us): those stay here.
    if K % 8 or (M % 8 and M < 128 and N % 8 == 0):
        return False
    if N % 8 and N < 256 and (N < 16 or M < 8192):
        return False  # few classes: padding them pays where the rows are many
    return 2 * M * N * K >= _MIN_WORK


def matmul(a, b):
    if b.ndim != 2 or a.ndim < 2 or a.dtype != torch.bfloat16 or b.dtype != torch.bfloat16:
        return None
    lead = a.shape[:-1]
    a2 = a.reshape(-1, a.shape[-1])
    if not _qualifies(a2, b):
        return None
    out = GemmFn.apply(a2, b, None, None, None)
    return out.reshape(tuple(lead) + (b.shape[1],))


def _grad_target(variable, w):
    """The fp32 parameter to accumulate the weight gradient into: only when ``w`` is the variable's bf16 shadow read."""
    p = getattr(variable, "_value", None)
    if not _WGRAD_IN_PLACE or variable is None or p is None or getattr(variable, "_shadow", None) is None or not p.requires_grad or p.dtype != torch.float32 or w.dtype != torch.bfloat16:
        return None
    if getattr(variable, "_shard_slices", None) is not None or p.numel() != w.numel():
        return None
    return p


def dense(x, kernel, bias, activation_name, kernel_shape=None, value=None):
    """Returns ``(output, activation_applied)`` or ``None``.  ``kernel`` may be a ``Variable`` (reshaped to the 2-D ``kernel_shape`` when
    given) or a tensor; ``value``: what the ``Variable`` reads as, when the caller has already read it."""
    from keras_b200.core.variables import Variable

    w = (kernel.value if value is None else value) if isinstance(kernel, Variable) else kernel
    if kernel_shape is not None:
        w = w.reshape(kernel_shape)
    if not isinstance(x, torch.Tensor) or x.dtype != torch.bfloat16 or w.dtype != torch.bfloat16 or w.ndim != 2 or x.ndim < 2:
        return None
    lead = x.shape[:-1]
    x2 = x.reshape(-1, x.shape[-1])
    if not _qualifies(x2, w):
        return None
    b = bias.value if isinstance(bias, Variable) else bias
    if b is not None and b.device != x.device:
        return None
    needs_grad = torch.is_grad_enabled() and (x2.requires_grad or w.requires_grad or (b is not None and b.requires_grad))
    if not needs_grad:
        name = {"gelu": "gelu_erf"}.get(activation_name, activation_name)
        act = _ACT.get(name)
        fused_act = act is not None
        N = w.shape[1]
        b32 = _bias_operand(b)
        if N % 8:
            w = kops.pad_columns(w, padded_width(N))
            b32 = torch.nn.functional.pad(b32, (0, w.shape[1] - N)) if b32 is not None else None
        out = gemm(x2, w, 0, 1, x2.shape[0], w.shape[1], x2.shape[1], bias=b32, act=act or 0)
        if N % 8:
            out = out[:, :N]
        return out.reshape(tuple(lead) + (N,)), fused_act
    target = _grad_target(kernel, w) if isinstance(kernel, Variable) else None
    bias_target = _grad_target(bias, b) if isinstance(bias, Variable) else None
    # relu, silu and gelu come with the product: their derivative is taken together with the bias gradient
    act = {"relu": 1, "silu": 3, "swish": 3, "gelu": 4}.get(activation_name, 0) if w.shape[1] % 8 == 0 else 0
    out = GemmFn.apply(x2, w, b, target, bias_target, act)
    return out.reshape(tuple(lead) + (w.shape[1],)), act != 0 or activation_name in (None, "linear")
