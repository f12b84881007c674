"""Calls of stock layers in inference, made straight from the graph's executor.

A layer call is some forty microseconds of Python around one or two launches: argument conversion, input spec, call context, scopes,
masks, and a cast of every weight it reads.  Where no gradient is recorded and the layer is a stock one, called on its inputs alone,
none of that can change the result, and the functions here go from the layer's attributes to the kernel.  Nothing is kept
between calls: each reads the attributes, the variables and the masks anew, and returns ``None`` (the layer is then called in the ordinary
way) when anything is out of the ordinary.  Weights stay float32; the product rounds them on their way in (``csrc/gemm_rows.cu``).
"""

import ctypes
import weakref

import torch

from keras_b200 import activations
from keras_b200.core import global_state
from keras_b200.core.keras_tensor import KerasTensor
from keras_b200.core.variables import Variable, get_stateless_scope
from keras_b200.kernels import attention as kattention
from keras_b200.kernels import dispatch
from keras_b200.kernels import gemm as kgemm
from keras_b200.kernels import ops as kops
from keras_b200.layers import layer as layer_module
from keras_b200.layers.attention.attention_layers import GroupedQueryAttention, MultiHeadAttention
from keras_b200.layers.core.dense import Dense
from keras_b200.layers.core.einsum_dense import EinsumDense
from keras_b200.layers.core.embedding import Embedding
from keras_b200.layers.layer import Layer
from keras_b200.layers.merging.merging_layers import Add, Multiply
from keras_b200.layers.normalization.normalization_layers import LayerNormalization, RMSNormalization

_BF16, _F32 = torch.bfloat16, torch.float32
_SINGLE_POLICIES = layer_module._SINGLE_POLICIES
# act codes of the GEMM's epilogue, by identity: a user's own function may well be called "gelu"
_EPILOGUE = {None: 0, activations.linear: 0, activations.relu: 1, activations.silu: 3, activations.gelu: 4}

# what a stock layer runs: a class whose method was replaced since is called in the ordinary way
_METHODS = [(Layer, "__call__"), (Layer, "_eager_call"), (Layer, "_set_output_mask")] + [
    (c, m) for c in (Dense, EinsumDense, Embedding, Add, Multiply, LayerNormalization, RMSNormalization, MultiHeadAttention, GroupedQueryAttention)
    for m in ("__call__", "call", "compute_mask")] + [
    (MultiHeadAttention, m) for m in ("_attend", "_compute_attention", "_attend_padded", "_takes_padding", "_compute_attention_mask")] + [
    (GroupedQueryAttention, m) for m in ("_compute_attention", "_compute_attention_mask")] + [(Add, "_merge_function"), (Multiply, "_merge_function")]
_STOCK = [getattr(c, m) for c, m in _METHODS]

_ATTRIBUTES = ("distribution", "tp_sequence_parallel", "tp_local_shards", "symbolic_scope")


def usable(x):
    """Whether layers of this call of a graph may be computed outside their own calls: nothing traces, redirects or distributes it.  Whether
    gradients are recorded is the caller's question: all of this module but ``add_norm`` is for calls without."""
    return (type(x) is torch.Tensor and x.is_cuda and x.device.index == torch.cuda.current_device()
            and not layer_module._NVTX_RANGES and get_stateless_scope() is None
            and all(global_state.get_global_attribute(a) is None for a in _ATTRIBUTES)
            and not torch._C._len_torch_function_stack() and not torch._C._len_torch_dispatch_stack()
            and not torch.is_autocast_enabled("cuda") and not torch.compiler.is_compiling() and torch._C._get_tracing_state() is None
            and all(getattr(c, m) is f for (c, m), f in zip(_METHODS, _STOCK)))


# ------------------------------------------------------------------------------------------------ launches
_SIGNED = set()


def _function(name, argtypes):
    fn = getattr(kops._lib(), name)
    if name not in _SIGNED:
        fn.argtypes = argtypes
        fn.restype = ctypes.c_int
        _SIGNED.add(name)
    return fn


_V, _I, _L = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
_DENSE = [_V] * 7 + [_I] * 3 + [_V] * 2 + [_I] * 2 + [_L] * 2 + [_I] * 5 + [_V] * 2
_ACTIVATION = {3: torch.nn.functional.silu, 4: torch.nn.functional.gelu}


def _product(x, weights, biases, act, as_layers=False):
    """``act(x @ [w0 w1 w2] + bias)`` of contiguous matrices of one type, as rows of a pitch that is a multiple of 8; ``None`` where the kernels do not
    take it.  ``as_layers``: with every bit of the layers' own calls, which see a layer's first call and whatever is not taken here: the
    products that those leave to the library (whose sums run along K as these do) are rounded before the bias and the activation."""
    K = x.shape[-1]
    if len(weights) == 1:
        widths = (weights[0].numel() // K,) if K else (0,)
        N = widths[0]
    else:
        widths = [w.numel() // K for w in weights] if K else [0]
        N = sum(widths)
        if any(n % 64 for n in widths) or any(w.dtype != weights[0].dtype for w in weights):
            return None
    M, fp32 = x.numel() // K if K else 0, weights[0].dtype == _F32
    # fewer than 64 columns of either operand: below a box of the copies, and nothing to gain
    if (M == 0 or K < 64 or K % 8 or N < 64 or not x.is_contiguous() or x.data_ptr() % 16 or M * N >= 1 << 40 or M >= 1 << 31
            or N % 8 and N < 256):  # few classes: the library's result is contiguous
        return None
    # Few rows: weights as they are stored.  A CTA has 64 columns and walks all of K, at a microsecond a block of 64: with three CTAs for every second
    # SM that is the weights' traffic ([77, 4096, 14336] 80 us, a weight placed and multiplied 82), with fewer up to 1024 of K a wait that costs no more
    # than the launch it saves ([77, 768, 768] 14 and 9 us); [77, 3072, 768] 48 and 19.
    rows = M <= 128 and (K <= 1024 or N > 96 * kgemm._sm_count(x.device))
    plain, bias16, apart, w, b = not fp32 and len(weights) == 1 and N % 8 == 0, False, False, [0, 0, 0], [0, 0, 0]  # plain: a matrix as the products read it
    for i, t in enumerate(weights):
        w[i] = t.data_ptr()
        if t.device != x.device or not t.is_contiguous() or not rows and w[i] % 16:
            return None
    biased = any(t is not None for t in biases)
    if as_layers:
        own = [kgemm.takes(M, n, K) for n in widths]
        apart = (biased or act > 1) and not own[0]
        if any(own) != all(own) and (biased or act > 1) or apart and N % 8:
            return None
    if biased:
        kinds = {t.dtype for t in biases if t is not None}
        if len(kinds) > 1 or not kinds <= {_F32, _BF16} or not all(t is None or t.is_contiguous() and t.device == x.device for t in biases):
            return None
        bias16 = kinds == {_BF16}
        if plain and not bias16:  # a bias is read in the layer's type wherever it is read
            biases, bias16 = [biases[0].to(_BF16)], True
        elif bias16 and (len(weights) > 1 or N % 8):  # these are placed beside one another, in float32
            biases, bias16 = [t if t is None else t.float() for t in biases], False
        for i, t in enumerate(biases):
            b[i] = t.data_ptr() if t is not None else 0
    n = (*widths, 0, 0)[:3]
    pitch = (N + 7) // 8 * 8 if rows else kgemm.padded_width(N)
    out = torch.empty((M, pitch), dtype=_BF16, device=x.device)
    scratch = None if rows or plain else torch.empty(K * pitch + 2 * pitch, dtype=_BF16, device=x.device)
    code = _function("kb200_dense_infer", _DENSE)(x.data_ptr(), *w, *b, *n, out.data_ptr(), scratch.data_ptr() if scratch is not None else None, M, K, K, pitch,
                                                  1 if fp32 else 0, 1 if bias16 else 0, 0 if apart and act > 1 else act, 1 if rows else 0, 1 if apart else 0,
                                                  kgemm._err_flag(x.device).data_ptr(), kops._stream())
    kops._check(code, "dense_infer")
    return _ACTIVATION[act](out) if apart and act > 1 else out


_NORM = [_V] * 8 + [_L, _I, ctypes.c_float, _I, _I, _I, _V]


def _normalise(x, residual, gamma, beta, eps, rms, narrow):
    """``(norm(x + residual), x + residual)`` over the last axis of contiguous bf16 tensors."""
    D = x.shape[-1]
    y = torch.empty_like(x)
    total = torch.empty_like(x) if residual is not None else None
    code = _function("kb200_norm_fwd", _NORM)(x.data_ptr(), residual.data_ptr() if residual is not None else None, total.data_ptr() if total is not None else None,
                                              gamma.data_ptr() if gamma is not None else None, beta.data_ptr() if beta is not None else None, y.data_ptr(), None, None,
                                              x.numel() // D, D, eps, 1 if rms else 0, 1 if narrow else 0, 1, kops._stream())
    kops._check(code, "norm_fwd")
    return y, total


# ------------------------------------------------------------------------------------------------ what a call may rely on
def _ordinary(layer):
    """A built layer in bf16 that was called before, with nothing around its own computation."""
    d = layer.__dict__
    policy = d["_dtype_policy"]
    return ("call" not in d and "__call__" not in d and d["built"] and d["_called"] and d["_remat_mode"] is None
            and d["activity_regularizer"] is None and type(policy) in _SINGLE_POLICIES and policy.compute_dtype == "bfloat16" and policy.quantization_mode is None
            and not d.get("_is_quantized") and not d.get("_calibrated") and len(d["_call_context_args"]) == 1)


def _input(layer, x):
    """The input in the layer's type where its shape passes the layer's checks, else ``None``."""
    if type(x) is not torch.Tensor or not x.is_cuda or x.get_device() != dispatch._current_device():
        return None
    if x.dtype != _BF16:
        if not x.dtype.is_floating_point or not layer.__dict__["autocast"] or not layer.__dict__["_convert_input_args"]:
            return None
        mask = getattr(x, "_keras_mask", None)
        x = x.to(_BF16)
        if mask is not None:
            return None  # the ordinary call knows whether the mask outlives the cast
    spec = layer.__dict__["_input_spec"]
    if spec is not None:
        seen = (id(spec), x.shape, x.dtype)
        if layer.__dict__.get("_spec_checked") != seen:
            try:
                layer_module.assert_input_compatibility(spec, x, layer.name)
            except Exception:
                return None  # the ordinary call raises it
            layer.__dict__["_spec_checked"] = seen
    return x


def _stored(variable):
    """What a variable holds, as the kernels read it: the parameter, or its bf16 shadow; ``None`` for anything else."""
    if type(variable) is not Variable or variable._shard_slices is not None or not variable._autocast:
        return None
    value = variable._value
    if value is None or not value.is_cuda or value.dtype not in (_F32, _BF16):
        return None
    shadow = variable._shadow
    if shadow is not None and shadow[0] == _BF16 and value.dtype == _F32:
        return shadow[1](value)
    return value


def _pass_mask(out, mask):
    if mask is not None:
        out._keras_mask = mask
    return out


# ------------------------------------------------------------------------------------------------ layers
def _matrix_layer(layer):
    """``(weight, bias, activation code)`` of a Dense or a one-product EinsumDense, or ``None``."""
    d = layer.__dict__
    if not _ordinary(layer) or d["lora_enabled"] or not d["autocast"]:  # without it weights are read as they are stored
        return None
    act = _EPILOGUE.get(d["activation"]) if d["activation"] is None or d["activation"] in _EPILOGUE else None
    w = _stored(d.get("_kernel"))
    if w is None or act is None:
        return None
    bias = None
    if d["bias"] is not None:
        bias = _stored(d["bias"])
        if bias is None:
            return None
    return w, bias, act


def _dense(layer, x):
    x = _input(layer, x)
    parts = _matrix_layer(layer) if x is not None else None
    if parts is None or parts[0].ndim != 2 or parts[0].shape[0] != x.shape[-1] or x.ndim < 2:
        return None
    out = _product(x, [parts[0]], [parts[1]], parts[2], True)
    if out is None:
        return None
    n = parts[0].shape[1]
    if out.shape[1] != n:
        out = out[:, :n]
    return _pass_mask(out.reshape(x.shape[:-1] + (n,)), getattr(x, "_keras_mask", None))


def _norm_parts(layer, x):
    """``(gamma, beta, epsilon, rms, narrow)`` of a normalisation over the last axis, or ``None``; ``narrow``: its float32 parameters are read in bf16."""
    d = layer.__dict__
    if not _ordinary(layer) or x.ndim < 1 or not 0 < x.shape[-1] <= 8192 or x.numel() == 0 or not x.is_contiguous() or x.data_ptr() % 16:
        return None
    axis = d["axis"]
    axis = axis[0] if isinstance(axis, (list, tuple)) and len(axis) == 1 else axis
    if not isinstance(axis, int) or axis not in (-1, x.ndim - 1) or not isinstance(d["epsilon"], float):
        return None
    if type(layer) is RMSNormalization:
        gamma, beta, rms = d["scale"], None, True
    else:
        rms = bool(d["rms_scaling"])
        gamma, beta = d["gamma"] if d["scale"] or rms else None, d["beta"] if d["center"] and not rms else None
    out, narrow = [], False
    for v in (gamma, beta):
        t = v
        if v is not None:
            t = v._value if type(v) is Variable and v._shard_slices is None else None
            if t is None or t.device != x.device or t.ndim != 1 or t.shape[0] != x.shape[-1]:
                return None
            if t.dtype == _BF16 and not torch.is_grad_enabled():
                t = t.float()
            if t.dtype != _F32 or not t.is_contiguous() or t.data_ptr() % 16:
                return None
            narrow = narrow or v._autocast and d["autocast"]  # of one layer all or none: a parameter in bf16 stays what it is
        out.append(t)
    return out[0], out[1], d["epsilon"], rms, narrow


def _carries_mask(layer):
    """RMSNormalization knows no masks: the ordinary call warns that one is lost."""
    return bool(layer.__dict__["_supports_masking"])


def _norm(layer, x):
    x = _input(layer, x)
    parts = _norm_parts(layer, x) if x is not None else None
    mask = getattr(x, "_keras_mask", None)
    if parts is None or mask is not None and not _carries_mask(layer):
        return None
    return _pass_mask(_normalise(x, None, *parts)[0], mask)


def _merge_inputs(layer, inputs):
    d = layer.__dict__
    if not _ordinary(layer) or not d["autocast"] or d["_reshape_required"] or d["_input_spec"] is not None or len(inputs) != 2:
        return None
    a, b = inputs
    if type(a) is not torch.Tensor or type(b) is not torch.Tensor or a.dtype != _BF16 or b.dtype != _BF16 or a.shape != b.shape or not a.is_cuda or b.device != a.device:
        return None
    m, n = getattr(a, "_keras_mask", None), getattr(b, "_keras_mask", None)
    if m is None or n is None:
        m = None  # as the layer has it: a mask that not every input has is none
    elif m.dtype != torch.bool or n.dtype != torch.bool or m.shape != n.shape:
        return None
    elif m is not n:
        m = torch.logical_or(m, n)
    return a, b, m


def _add(layer, inputs):
    parts = _merge_inputs(layer, inputs)
    return None if parts is None else _pass_mask(torch.add(parts[0], parts[1]), parts[2])


def _multiply(layer, inputs):
    parts = _merge_inputs(layer, inputs)
    return None if parts is None else _pass_mask(torch.mul(parts[0], parts[1]), parts[2])


def add_norm(add, norm, inputs):
    """``(sum, norm(sum))`` of an Add and of a normalisation that reads it, from one pass; ``None`` where they run by themselves."""
    parts = _merge_inputs(add, inputs)
    if parts is None:
        return None
    a, b, mask = parts
    if not (a.is_contiguous() and b.is_contiguous()) or b.data_ptr() % 16 or _input(norm, a) is None or mask is not None and not _carries_mask(norm):
        return None
    how = _norm_parts(norm, a)
    if how is None:
        return None
    if torch.is_grad_enabled():
        if type(norm) is not LayerNormalization:  # its parameters are float32 leaves; those of RMSNormalization are read in the layer's type
            return None
        total, y = kops.FusedAddNorm.apply(a, b, *how[:4])
    else:
        y, total = _normalise(a, b, *how)
    return _pass_mask(total, mask), _pass_mask(y, mask)


_EMBED = [_V] * 3 + [_L, _I, _L] + [_I] * 4 + [_V]


def _embedding(layer, ids):
    d = layer.__dict__
    if not _ordinary(layer) or d["lora_enabled"] or d["_input_spec"] is not None or type(ids) is not torch.Tensor or not ids.is_cuda or ids.get_device() != dispatch._current_device():
        return None
    if ids.dtype not in (torch.int32, torch.int64) or getattr(ids, "_keras_mask", None) is not None or ids.numel() == 0:
        return None
    table = _stored(d.get("_embeddings"))
    if table is None or table.device != ids.device or table.ndim != 2 or table.shape[1] % 8 or not table.is_contiguous() or table.data_ptr() % 16 or not ids.is_contiguous():
        return None
    V, D = table.shape
    out = torch.empty(ids.shape + (D,), dtype=_BF16, device=ids.device)
    code = _function("kb200_embedding_fwd", _EMBED)(table.data_ptr(), ids.data_ptr(), out.data_ptr(), ids.numel(), D, V, 1 if table.dtype == _BF16 else 0, 1,
                                                    1 if ids.dtype == torch.int32 else 0, 1, kops._stream())
    kops._check(code, "embedding_fwd")
    return _pass_mask(out, torch.ne(ids, 0) if d["mask_zero"] else None)


def _attention(layer, x, causal, mask=None):
    """Self-attention of a stock layer: three projections as one product, the attention kernel, the output projection.  ``mask``: of rows and
    keys, where the call names one; else what the input carries."""
    d = layer.__dict__
    x = _input(layer, x)
    grouped = type(layer) is GroupedQueryAttention
    if x is None or x.ndim != 3 or not _ordinary(layer) or d["_input_spec"] is not None or d["_flash_attention"] is False:
        return None
    if grouped:
        if d["dropout"] != 0.0 or d["use_gate"]:
            return None
        heads, kv, size, scale = d["num_query_heads"], d["num_key_value_heads"], d["head_dim"], d["_inverse_sqrt_head_dim"]
    else:
        if d["_dropout"] != 0.0 or d["_use_gate"] or tuple(d["_attention_axes"]) != (1,) or d["_sliding_window"] is not None or d["_value_dim"] != d["_key_dim"]:
            return None
        heads = kv = d["_num_heads"]
        size, scale = d["_key_dim"], d["_inverse_sqrt_key_dim"]
    if mask is None:
        mask = getattr(x, "_keras_mask", None)
    elif type(mask) is not torch.Tensor:
        return None
    if size not in (64, 128) or mask is not None and (grouped or causal or mask.dtype != torch.bool or mask.ndim != 2 or mask.shape != x.shape[:2] or mask.stride(1) != 1):
        return None
    parts = []
    for sub in (d["_query_dense"], d["_key_dense"], d["_value_dense"], d["_output_dense"]):
        if type(sub) is not EinsumDense or not _sub_ordinary(sub):
            return None
        p = _matrix_layer(sub)
        if p is None or p[2] != 0:
            return None
        parts.append(p)
    if any(sub.__dict__["_gemm"] != (1, 2) for sub in (d["_query_dense"], d["_key_dense"], d["_value_dense"])) or d["_output_dense"].__dict__["_gemm"] != (2, 1):
        return None
    K = x.shape[-1]
    if [tuple(p[0].shape) for p in parts[:3]] != [(K, heads, size), (K, kv, size), (K, kv, size)] or tuple(parts[3][0].shape[:2]) != (heads, size):
        return None
    if any(p[1] is not None and tuple(p[1].shape) != tuple(p[0].shape[1:]) for p in parts[:3]) or parts[3][1] is not None and parts[3][1].ndim != 1:
        return None
    if kattention.os.environ.get("KERAS_B200_FLASH_ATTENTION", "inference") == "0":
        return None
    qkv = _product(x, [p[0] for p in parts[:3]], [p[1] for p in parts[:3]], 0, True)
    if qkv is None:
        return None
    B, T = x.shape[:2]
    qkv = qkv.view(B, T, heads + 2 * kv, size)
    q, k, v = qkv[:, :, :heads], qkv[:, :, heads:heads + kv], qkv[:, :, heads + kv:]
    if mask is not None:
        out = kattention.flash_attention(q, k, v, mask[:, None, None, :], scale, False, row_mask=mask)
    else:
        out = kattention.flash_attention(q, k, v, None, scale, causal)
    if out is None:
        return None
    out = _product(out.view(B, T, heads * size), [parts[3][0]], [parts[3][1]], 0, True)
    return None if out is None else _pass_mask(out[:, :parts[3][0].shape[2]].view(B, T, -1), mask)


def joint_projections(layer, x):
    """Query, key and value of a self-attention layer's call with gradients from one launch each way, or ``None``."""
    d = layer.__dict__
    if type(x) is not torch.Tensor or x.dtype != _BF16 or x.ndim != 3 or not torch.is_grad_enabled() or not dispatch.enabled(x) or not usable(x) or not _ordinary(layer):
        return None
    subs = [d["_query_dense"], d["_key_dense"], d["_value_dense"]]
    for sub in subs:
        s = sub.__dict__
        if (type(sub) is not EinsumDense or not _ordinary(sub) or s["_input_spec"] is not None or s["lora_enabled"] or s["_gemm"] != (1, 2)
                or not (s["activation"] is None or s["activation"] is activations.linear) or type(s.get("_kernel")) is not Variable
                or s["_kernel"]._shard_slices is not None or s["_kernel"].shape[0] != x.shape[-1]):
            return None
    biases = [sub.__dict__["bias"] for sub in subs]
    if all(b is None for b in biases):
        biases = []
    elif any(type(b) is not Variable or tuple(b.shape) != tuple(sub.__dict__["_kernel"].shape[1:]) for b, sub in zip(biases, subs)):
        return None
    kernels = [sub.__dict__["_kernel"] for sub in subs]
    weights = [k.value for k in kernels]  # in the layer's type: its call has set the scope
    if any(w.dtype != _BF16 or w.ndim != 3 for w in weights) or not (x.requires_grad or any(w.requires_grad for w in weights)):
        return None
    return kgemm.projections(x, kernels, biases, weights)


def _sub_ordinary(layer):
    """A projection inside an attention layer: called by that layer with tensors it has made, so the specs of its inputs hold."""
    return layer.__dict__["_input_spec"] is None


# ------------------------------------------------------------------------------------------------ the graph
class _Plan:
    """What was found in a graph.  It lives in the graph, and so no longer than the layers: one that was kept beside it held their weights until
    a collection after the one that took the graph.  A copied or pickled graph has other layers, and none."""

    __slots__ = ("nodes", "runs", "pairs", "__weakref__")

    def __init__(self, nodes):
        self.nodes = nodes
        self.runs, self.pairs = _build_plan(nodes)

    def __deepcopy__(self, memo):
        return None

    def __reduce__(self):
        return type(None), ()


_PLANS = weakref.WeakValueDictionary()  # the plans in use, by the graph's identity: clearing it has them made anew


def plan_of(function, nodes):
    plan = function.__dict__.get("_direct_plan")
    if plan is None or plan.nodes is not nodes or _PLANS.get(id(function)) is not plan:
        plan = function.__dict__["_direct_plan"] = _PLANS[id(function)] = _Plan(nodes)
    return plan.runs, plan.pairs


def _build_plan(nodes):
    """``{id(node): run}`` with ``run(env)`` the output of that node's call or ``None``, and ``{id(add node): (norm node, inputs)}`` of the pairs
    that one pass computes."""
    runs, pairs = {}, {}
    readers = {}
    for n in nodes:
        for t in n.input_tensors:
            readers.setdefault(id(t), []).append(n)
    for n in nodes:
        op, a = n.operation, n.arguments
        kind = type(op)
        given = {k: v for k, v in a.kwargs.items() if v is not None}
        if len(n.outputs) != 1:
            continue
        if kind in (Dense, LayerNormalization, RMSNormalization, Embedding) and len(a.args) == 1 and isinstance(a.args[0], KerasTensor) and not given:
            run = {Dense: _dense, Embedding: _embedding}.get(kind, _norm)
            runs[id(n)] = lambda env, op=op, t=id(a.args[0]), run=run: run(op, env[t])
        elif kind in (Add, Multiply) and len(a.args) == 1 and isinstance(a.args[0], (list, tuple)) and len(a.args[0]) == 2 and not given and all(
                isinstance(t, KerasTensor) for t in a.args[0]):
            ids = tuple(id(t) for t in a.args[0])
            run = _add if kind is Add else _multiply
            runs[id(n)] = lambda env, op=op, ids=ids, run=run: run(op, (env[ids[0]], env[ids[1]]))
            if kind is Add:
                for r in readers.get(id(n.outputs[0]), []):
                    if type(r.operation) in (LayerNormalization, RMSNormalization) and len(r.input_tensors) == 1 and len(r.outputs) == 1 and len(r.arguments.args) == 1 and all(
                            v is None for v in r.arguments.kwargs.values()):
                        pairs[id(n)] = (r, ids)
                        break
        elif kind in (MultiHeadAttention, GroupedQueryAttention) and len(a.args) == 2 and a.args[0] is a.args[1] and isinstance(a.args[0], KerasTensor):
            causal, mask = given.pop("use_causal_mask", False), given.pop("query_mask", None)
            if not isinstance(causal, bool) or given.pop("value_mask", None) is not mask or given or not (mask is None or isinstance(mask, KerasTensor)):
                continue
            runs[id(n)] = lambda env, op=op, t=id(a.args[0]), causal=causal, m=None if mask is None else id(mask): _attention(
                op, env[t], causal, None if m is None else env[m])
    return runs, pairs
