"""Graph-level fusion for ``Functional`` models.

The executor of a ``Functional`` walks its nodes in order; this module finds, once per model,
the node patterns that a single sm_100a kernel can execute:

* ``BatchNormalization → ReLU`` (or ReLU6)              → BN apply with fused ReLU
* ``BatchNormalization → Add(other) [→ ReLU]``          → BN apply with fused residual add (and ReLU)

(the residual bottleneck of keras/src/applications/resnet.py:219-273 is conv→BN→ReLU ×2, conv→BN,
Add, ReLU).  A fused BN is *deferred*: its node records the input, and the kernel runs when the
consumer node is reached so the residual operand is available.  Patterns only fire on CUDA tensors
with a channels-last BN; otherwise execution is node by node as written.
"""

import math
import threading

import torch

from keras_b200 import activations
from keras_b200.layers.activations.activation_layers import Activation, ReLU
from keras_b200.layers.merging.merging_layers import Add
from keras_b200.layers.normalization.normalization_layers import BatchNormalization


class Deferred:
    __slots__ = ("layer", "x", "pre_bias", "stats", "shape", "dtype", "device", "ndim")

    def __init__(self, layer, x, pre_bias=None, stats=None):
        self.layer, self.x, self.pre_bias, self.stats = layer, x, pre_bias, stats
        self.shape, self.dtype, self.device, self.ndim = x.shape, x.dtype, x.device, x.ndim


class Padded:
    """Input of a folded ZeroPadding2D: the consumer applies ``pairs`` itself."""

    __slots__ = ("x", "pairs")

    def __init__(self, x, pairs):
        self.x, self.pairs = x, pairs


class NoBias:
    """Output of a convolution whose bias add was folded into the following BatchNormalization."""

    __slots__ = ("x", "bias", "stats")

    def __init__(self, x, bias, stats=None):
        self.x, self.bias, self.stats = x, bias, stats


def _plain(node, *types):
    """Whether a node is its stock layer and nothing more, so that a kernel may stand for the whole call: the exact class (a subclass may
    compute anything), called on its inputs alone (a BatchNormalization may have been told its ``training``), with no regularizer of
    its output to report and its input cast as the policy says."""
    op, arguments = node.operation, node.arguments
    return (type(op) in types and "call" not in vars(op) and op.activity_regularizer is None and op.autocast and len(arguments.args) == 1
            and all(v is None for v in arguments.kwargs.values()))


def _rectifier_bound(node):
    """Upper bound of a rectifier layer (infinity for a plain one, six with the strict derivative of the library's ``relu6``), or ``None``."""
    op = node.operation
    if not _plain(node, ReLU, Activation):
        return None
    if isinstance(op, Activation):  # by identity: a user's own function may well be called "relu"
        return math.inf if op.activation is activations.relu else 6.0 if op.activation is activations.relu6 else None
    if op.negative_slope != 0.0 or op.threshold != 0.0:
        return None
    return math.inf if op.max_value is None else 6.0 if op.max_value == 6.0 else None


def relu_cap(op):
    """Upper bound of a layer that ``build_plan`` took for a rectifier, or ``None``."""
    return None if (op.max_value is None if isinstance(op, ReLU) else op.activation is activations.relu) else 6.0


def build_plan(function):
    """Return {id(node): role} with roles 'defer_bn', 'consume_add', 'consume_relu', 'maybe_identity'."""
    nodes = function._ordered_nodes()
    in_graph = set(id(n) for n in nodes)
    consumers = {}
    for n in nodes:
        for t in n.input_tensors:
            consumers.setdefault(id(t), []).append(n)
    output_ids = {id(t) for t in function._outputs}
    plan = {}
    for n in nodes:
        op = n.operation
        if not _plain(n, BatchNormalization) or op.renorm or op.synchronized or len(n.outputs) != 1:
            continue
        out = n.outputs[0]
        if id(out) in output_ids:
            continue
        cons = consumers.get(id(out), [])
        if len(cons) != 1:
            continue
        c = cons[0]
        if getattr(c.operation, "compute_dtype", None) != op.compute_dtype:
            continue  # the consumer casts first
        if plan.get(id(c)) in ("consume_add", "consume_add_relu"):
            # second BN operand of an already planned Add: deferred too, so that its producing convolution can
            # drop its bias; the executor materialises it before the fused BN+Add of the first operand
            plan[id(n)] = "defer_bn"
            continue
        if id(c) in plan:
            continue
        if _rectifier_bound(c) is not None and len(c.input_tensors) == 1:
            plan[id(n)] = "defer_bn"
            plan[id(c)] = "consume_relu"
        elif _plain(c, Add) and len(c.input_tensors) == 2 and len(c.outputs) == 1:
            other = [t for t in c.input_tensors if t is not out]
            if len(other) != 1 or tuple(other[0].shape) != tuple(out.shape):
                continue
            plan[id(n)] = "defer_bn"
            plan[id(c)] = "consume_add"
            add_out = c.outputs[0]
            cc = consumers.get(id(add_out), [])
            if (id(add_out) not in output_ids and len(cc) == 1 and _rectifier_bound(cc[0]) == math.inf and id(cc[0]) not in plan
                    and cc[0].operation.compute_dtype == op.compute_dtype):
                plan[id(c)] = "consume_add_relu"
                plan[id(cc[0])] = "identity"
    # Convolution bias feeding a fused BN: the normalised output does not depend on it (training
    # mode) and its gradient is exactly zero, so the add and the bias-gradient reduction are dropped;
    # the bias only enters the moving-mean update (and the shift in inference mode).
    from keras_b200.layers.convolutional.base_conv import Conv1D, Conv2D, Conv3D

    producers = {}
    for n in nodes:
        for t in n.outputs:
            producers[id(t)] = n
    for n in nodes:
        if plan.get(id(n)) != "defer_bn":
            continue
        src = producers.get(id(n.input_tensors[0]))
        if src is None or id(src) in plan:
            continue
        op = src.operation
        if not _plain(src, Conv1D, Conv2D, Conv3D) or op.lora_enabled or op.data_format != "channels_last":
            continue
        if op.activation is not None and op.activation is not activations.linear:
            continue
        out = src.outputs[0]
        if id(out) in output_ids or len(consumers.get(id(out), [])) != 1 or len(src.input_tensors) != 1:
            continue
        if n.operation.axis % len(out.shape) != len(out.shape) - 1:
            continue
        plan[id(src)] = "conv_fold_bias"
    # ZeroPadding2D in front of a max pooling or of a bias-folded convolution ("valid" padding): the padded copy
    # is never made; the pooling kernel and the convolution take the padding as a parameter.
    from keras_b200.layers.pooling.pooling import MaxPooling2D
    from keras_b200.layers.reshaping.reshaping_layers import ZeroPadding2D

    for n in nodes:
        op = n.operation
        if not _plain(n, ZeroPadding2D) or op.data_format != "channels_last" or id(n) in plan or len(n.input_tensors) != 1:
            continue
        out = n.outputs[0]
        cons = consumers.get(id(out), [])
        if id(out) in output_ids or len(cons) != 1:
            continue
        c = cons[0]
        cop = c.operation
        if _plain(c, MaxPooling2D) and cop.padding == "valid" and cop.data_format == "channels_last" and id(c) not in plan:
            plan[id(n)] = "pad_fold"
            plan[id(c)] = "pool_padded"
        elif plan.get(id(c)) == "conv_fold_bias" and cop.rank == 2 and cop.padding == "valid" and all(lo == hi for lo, hi in op.padding):
            plan[id(n)] = "pad_fold"
    # Activations read by exactly two consumers that can share one gradient buffer (kernels/grad_merge.py): a bias-folded
    # convolution reading the tensor itself, plus either a second such convolution (projection shortcut) or the fused
    # BatchNorm+Add that takes the tensor as its residual operand (identity shortcut).
    merge = set()
    for n in nodes:
        for out in n.outputs:
            cons = consumers.get(id(out), [])
            if id(out) in output_ids or len(cons) != 2 or cons[0] is cons[1]:
                continue
            kinds = []
            for c in cons:
                role = plan.get(id(c))
                if role == "conv_fold_bias" and len(c.input_tensors) == 1:
                    kinds.append("conv")
                elif role in ("consume_add", "consume_add_relu"):
                    # the residual operand is the one that does not come from a deferred BatchNormalization
                    src = producers.get(id(out))
                    if src is not None and plan.get(id(src)) != "defer_bn":
                        kinds.append("add")
            if sorted(kinds) in (["conv", "conv"], ["add", "conv"]):
                merge.add(id(out))
    plan["merge_tensors"] = merge
    return plan


def run_pool_padded(layer, x, pairs):
    from keras_b200 import ops
    from keras_b200.kernels import dispatch

    out = dispatch.max_pool2d(x, layer.pool_size, layer.strides, "valid", zero_pad=pairs)
    if out is not None:
        return out
    pads = [(0, 0), tuple(pairs[0]), tuple(pairs[1]), (0, 0)]
    return layer(ops.pad(x, pads))


class RecordedInputs(threading.local):
    """The batch of a step that is being recorded in this thread.  Its cast to bf16 is left to whoever copies a batch in, which reads
    it anyway: ``casts`` maps the place of a batch tensor to the bf16 tensor that the recorded step reads; ``read``: the places of those that
    a convolution was given as they are, or casts otherwise."""

    def __init__(self):
        self.end()

    def begin(self, leaves):
        self._leaves = [(leaf, leaf._version) if isinstance(leaf, torch.Tensor) else None for leaf in leaves]
        self.casts, self.read = {}, set()
        # Made before the recording: what is allocated during one may lie where an earlier kernel of the graph keeps something of its own,
        # which a replay writes there after the cast.
        self._room = [torch.empty_like(leaf, dtype=torch.bfloat16) if isinstance(leaf, torch.Tensor) and leaf.is_cuda and leaf.dtype == torch.float32 else None
                      for leaf in leaves]

    def end(self):
        made = getattr(self, "casts", None), getattr(self, "read", None)
        self._leaves, self._room, self.casts, self.read = (), (), {}, set()
        return made

    def given(self, x):
        """``x`` itself goes to a reader."""
        self.read.update(i for i, entry in enumerate(self._leaves) if entry is not None and entry[0] is x)
        return x

    def cast(self, x, dtype):
        for i, entry in enumerate(self._leaves):
            if entry is not None and entry[0] is x and entry[1] == x._version and self._room[i] is not None and dtype == torch.bfloat16:
                return self.casts.setdefault(i, self._room[i])
        return None


recorded_inputs = RecordedInputs()


def shared_cast(layer, x, casts):
    """``x`` in the layer's compute dtype, cast once for all the convolutions of a pass that read it (the input of a block with a
    projected shortcut: [256, 56, 56, 256] in float32 is 185 us a cast).  Only where no gradient flows back, which would
    otherwise be summed in the narrow type; ``casts`` lives for one pass."""
    if not isinstance(x, torch.Tensor) or x.requires_grad or not x.dtype.is_floating_point:
        return recorded_inputs.given(x)
    td = layer._compute_torch_dtype()
    if x.dtype == td or not td.is_floating_point or (x.dtype == torch.float32 and x.shape[-1] % 8):
        return recorded_inputs.given(x)  # an fp32 input with few channels is cast inside the patch kernel
    kept = casts.get((id(x), td))
    if kept is None or kept[0] is not x:
        recorded = recorded_inputs.cast(x, td)
        kept = casts[(id(x), td)] = (x, recorded_inputs.given(x).to(td) if recorded is None else recorded)
    return kept[1]


def run_conv_nobias(layer, x, pairs=None, want_stats=False):
    """The convolution of ``layer`` without its bias add (autocast applied as ``Layer.__call__`` would).

    ``pairs``: symmetric zero padding of a folded ZeroPadding2D, applied by the convolution itself.
    Returns ``(y, stats)``; ``stats`` holds the per-channel partial sums of ``y`` left by the convolution kernel's
    epilogue when ``want_stats`` is set and that kernel ran (else ``None``)."""
    from keras_b200 import ops
    from keras_b200.core.variables import AutocastScope
    from keras_b200.kernels import conv as kconv

    td = layer._compute_torch_dtype()
    with AutocastScope(layer.compute_dtype):
        if layer.rank == 2 and layer.groups == 1 and type(layer).convolution_op is BaseConvOp():
            padding = layer.padding if pairs is None else tuple(lo for lo, _ in pairs)
            w = layer.kernel.value
            xin = x
            if xin.dtype != td and xin.dtype.is_floating_point and not (xin.dtype == torch.float32 and w.shape[-2] % 8):
                xin = xin.to(td)  # an fp32 input with few channels is cast inside the patch kernel
            out = kconv.conv(xin, w, layer.strides, padding, layer.data_format, layer.dilation_rate, grad_target=layer.kernel, want_stats=want_stats)
            if out is not None:
                return out if want_stats else (out, None)
        if x.dtype != td and x.dtype.is_floating_point:
            x = x.to(td)
        if pairs is None:
            return layer.convolution_op(x, layer.kernel), None
        return ops.conv(x, layer.kernel, strides=list(layer.strides), padding=tuple(lo for lo, _ in pairs),
                        dilation_rate=layer.dilation_rate, data_format=layer.data_format), None


def BaseConvOp():
    from keras_b200.layers.convolutional.base_conv import BaseConv

    return BaseConv.convolution_op


def applicable(x):
    return isinstance(x, torch.Tensor) and x.is_cuda


def run_bn(layer, x, training, residual=None, relu=False, pre_bias=None, stats=None, cap=None):
    """Execute a (possibly fused) BatchNormalization outside of ``Layer.__call__``."""
    from keras_b200.kernels import dispatch

    train = bool(training) and layer.trainable
    td = layer._compute_torch_dtype()
    if x.dtype != td and x.dtype.is_floating_point:
        x, stats = x.to(td), None
    if residual is not None and residual.dtype != td and residual.dtype.is_floating_point:
        residual = residual.to(td)
    if residual is not None and residual.shape != x.shape:  # the kernel adds element to element: a broadcast sum is made outside
        out = run_bn(layer, x, training, pre_bias=pre_bias, stats=stats) + residual
        return torch.relu(out) if relu else out
    bias_value = pre_bias._value if pre_bias is not None else None
    out = dispatch.batch_norm(layer, x, train, residual=residual, relu=relu, pre_bias=bias_value, conv_stats=stats, cap=cap)
    if out is not None:
        if pre_bias is not None and train:
            # A bias in front of a batch normalization in training mode is removed with the batch mean: its gradient is exactly
            # zero.  The fused kernel never materialises it, so the variable is marked: gradient storage reports a zero
            # gradient for it (the optimizer then treats it as the reference does, weight decay included) instead of none.
            pre_bias._gradient_is_zero_when_absent = True
        return out
    if pre_bias is not None:
        x = x + pre_bias.value.to(x.dtype)
    out = layer(x, training=training)
    if residual is not None:
        out = out + residual
    if relu:
        out = torch.relu(out) if cap is None else torch.nn.functional.hardtanh(out, 0.0, cap)
    return out
