"""Workloads whose speed is tracked, each a pass through the public API of the package.

Seven kinds of program, from the smallest call to the largest:

* ``mlp``      one ``train_on_batch`` step of a dense classifier under the default float32 policy (tabular data, digits)
* ``lm``       one ``train_on_batch`` step of a causal decoder: embedding, pre-norm attention and GELU MLP, vocabulary
               projection, cross-entropy, AdamW, under ``mixed_bfloat16`` (language-model training)
* ``infer``    logits of a causal decoder for a batch of prompts (scoring, prefill) in bfloat16, GPT-style or with
               grouped-query attention, RMS norm and a gated MLP
* ``encode``   token states of a post-norm encoder over padded batches, the padding masked by ``Embedding(mask_zero=True)``
               and set to zero in the result
* ``residual`` one ``train_on_batch`` step of two ResNet bottleneck blocks under a classifier of pixels, SGD with momentum
* ``mobile``   one ``train_on_batch`` step of two inverted residual blocks (depthwise convolutions) under the same classifier
* ``lstm``     one ``train_on_batch`` step of an LSTM regressor over whole sequences, float32

Training cases return the loss, the optimizer's first moments (which hold the step's gradients) and updated weights.
"""

import math

import torch

import keras_b200 as keras

_EPS = 1e-5


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # a digits classifier at the batch size users start with: the step is launches and little else
        {"name": "mlp_digits", "kind": "mlp", "batch": 128, "features": 784, "hidden": 512, "classes": 10},
        # two layers of the GPT-2 benchmark configuration at its own batch, length and vocabulary
        {"name": "lm_gpt2", "kind": "lm", "batch": 16, "seq": 1024, "d": 768, "heads": 12, "ffn": 3072, "vocab": 50257, "layers": 2},
        # a small model on text of uneven length: no dimension of the batch is a multiple of a tile
        {"name": "lm_ragged", "kind": "lm", "batch": 8, "seq": 333, "d": 512, "heads": 8, "ffn": 2048, "vocab": 8009, "layers": 2},
        # one short prompt: the latency of a forward pass
        {"name": "infer_prompt", "kind": "infer", "style": "gpt", "batch": 1, "seq": 77, "d": 768, "heads": 12, "kv_heads": 12, "ffn": 3072,
         "vocab": 50257, "layers": 2},
        # scoring of whole contexts with the GPT-2 configuration
        {"name": "infer_gpt2", "kind": "infer", "style": "gpt", "batch": 16, "seq": 1024, "d": 768, "heads": 12, "kv_heads": 12, "ffn": 3072,
         "vocab": 50257, "layers": 2},
        # one layer of the 8B decoder configuration at its own context length
        {"name": "infer_8b", "kind": "infer", "style": "gated", "batch": 2, "seq": 4096, "d": 4096, "heads": 32, "kv_heads": 8, "ffn": 14336,
         "vocab": 128256, "layers": 1},
        # many short texts through two layers of the 1.3B decoder configuration
        {"name": "infer_short", "kind": "infer", "style": "gpt", "batch": 64, "seq": 128, "d": 2048, "heads": 16, "kv_heads": 16, "ffn": 8192,
         "vocab": 50257, "layers": 2},
        # a batch of padded sentences through two encoder layers of the usual base size
        {"name": "encode_padded", "kind": "encode", "batch": 32, "seq": 384, "d": 768, "heads": 12, "ffn": 3072, "vocab": 30522, "layers": 2},
        # the 28x28 stage of ResNet-50 at the benchmark's batch, entered with a stride
        {"name": "residual_28", "kind": "residual", "batch": 256, "size": 56, "cin": 256, "width": 128, "stride": 2, "classes": 64},
        # a small batch of odd-sized images, channels that are no power of two
        {"name": "residual_odd", "kind": "residual", "batch": 24, "size": 35, "cin": 192, "width": 96, "stride": 2, "classes": 37},
        # the 28x28 stage of a MobileNet-style network
        {"name": "mobile_28", "kind": "mobile", "batch": 128, "size": 56, "cin": 24, "cout": 32, "expand": 6, "k": 3, "stride": 2, "classes": 21},
        # a forecaster over windows of a multivariate series
        {"name": "lstm_series", "kind": "lstm", "batch": 64, "steps": 100, "features": 32, "units": 256, "outputs": 8},
    ]


def _log(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, int(round(v / multiple)) * multiple)


def draw(rng):
    kind = rng.choice(["mlp", "lm", "lm", "infer", "infer", "infer", "encode", "encode", "residual", "residual", "mobile", "mobile", "lstm"])
    if kind == "mlp":
        return {"kind": kind, "batch": _log(rng, 16, 4096), "features": _log(rng, 16, 2048), "hidden": _log(rng, 64, 2048), "classes": _log(rng, 2, 100)}
    if kind in ("lm", "infer", "encode"):
        hd = rng.choice([64, 64, 128])
        heads = rng.choice([4, 6, 8, 12, 16])
        d = hd * heads
        ffn = rng.choice([2, 3, 4]) * d
        seq = _log(rng, 32, 2048)
        tokens = _log(rng, 256, 16384)
        case = {"kind": kind, "batch": max(1, tokens // seq), "seq": seq, "d": d, "heads": heads, "ffn": ffn, "vocab": _log(rng, 1000, 50000), "layers": 2}
        if kind == "infer":
            gated = rng.random() < 0.5
            case.update(style="gated" if gated else "gpt", kv_heads=heads // rng.choice([1, 2]) if gated else heads)
        return case
    if kind == "residual":
        size, cin, width = rng.choice([(56, 64, 64), (56, 256, 128), (28, 512, 256), (14, 1024, 512)])
        size = max(7, size + rng.randint(-3, 3))
        return {"kind": kind, "batch": _log(rng, 8, 192), "size": size, "cin": cin, "width": width, "stride": rng.choice([1, 2]), "classes": _log(rng, 2, 150)}
    if kind == "mobile":
        size, cin, cout = rng.choice([(112, 16, 24), (56, 24, 32), (28, 32, 64), (14, 96, 160)])
        size = max(7, size + rng.randint(-3, 3))
        return {"kind": kind, "batch": _log(rng, 8, 128 if size < 80 else 32), "size": size, "cin": cin, "cout": cout, "expand": rng.choice([4, 6]),
                "k": rng.choice([3, 3, 5]), "stride": rng.choice([1, 2]), "classes": _log(rng, 2, 150)}
    return {"kind": kind, "batch": _log(rng, 8, 256), "steps": _log(rng, 12, 160), "features": _log(rng, 4, 256), "units": _log(rng, 32, 512, 8),
            "outputs": _log(rng, 1, 32)}


# ------------------------------------------------------------------------------------------------ models
class _Positions(keras.layers.Layer):
    """Learned position table added to the token embeddings."""

    def build(self, input_shape):
        self.table = self.add_weight(shape=tuple(input_shape[1:]), initializer="zeros", name="table")

    def call(self, x):
        return x + keras.ops.cast(self.table, x.dtype)


def _decoder(c):
    L = keras.layers
    tokens = keras.Input((c["seq"],), dtype="int32")
    gated = c.get("style") == "gated"
    h = L.Embedding(c["vocab"], c["d"])(tokens)
    h = h if gated else _Positions()(h)
    hd = c["d"] // c["heads"]
    norm = (lambda: L.RMSNormalization(epsilon=_EPS)) if gated else (lambda: L.LayerNormalization(epsilon=_EPS))
    for _ in range(c["layers"]):
        a = norm()(h)
        if gated:
            a = L.GroupedQueryAttention(hd, c["heads"], c["kv_heads"], use_bias=False)(a, a, use_causal_mask=True)
        else:
            a = L.MultiHeadAttention(c["heads"], hd, use_bias=False)(a, a, use_causal_mask=True)
        h = L.Add()([h, a])
        m = norm()(h)
        if gated:
            m = L.Multiply()([L.Dense(c["ffn"], activation="silu", use_bias=False)(m), L.Dense(c["ffn"], use_bias=False)(m)])
            m = L.Dense(c["d"], use_bias=False)(m)
        else:
            m = L.Dense(c["d"])(L.Dense(c["ffn"], activation="gelu")(m))
        h = L.Add()([h, m])
    return keras.Model(tokens, L.Dense(c["vocab"], use_bias=False)(norm()(h)))


def _encoder(c):
    L = keras.layers
    tokens = keras.Input((c["seq"],), dtype="int32")
    h = L.Embedding(c["vocab"], c["d"], mask_zero=True)(tokens)
    for _ in range(c["layers"]):
        h = L.LayerNormalization(epsilon=_EPS)(L.Add()([h, L.MultiHeadAttention(c["heads"], c["d"] // c["heads"])(h, h)]))
        h = L.LayerNormalization(epsilon=_EPS)(L.Add()([h, L.Dense(c["d"])(L.Dense(c["ffn"], activation="gelu")(h))]))
    return keras.Model(tokens, h)


def _residual(c):
    L = keras.layers
    x = keras.Input((c["size"], c["size"], c["cin"]))
    w, s = c["width"], c["stride"]

    def conv(t, filters, k, stride=1):
        return L.BatchNormalization(epsilon=1.001e-5)(L.Conv2D(filters, k, strides=stride, padding="same", use_bias=False)(t))

    t = L.ReLU()(conv(x, w, 1, s))
    t = L.ReLU()(conv(t, w, 3))
    t = conv(t, 4 * w, 1)
    h = L.ReLU()(L.Add()([conv(x, 4 * w, 1, s), t]))
    t = L.ReLU()(conv(h, w, 1))
    t = L.ReLU()(conv(t, w, 3))
    h = L.ReLU()(L.Add()([h, conv(t, 4 * w, 1)]))
    return keras.Model(x, L.Dense(c["classes"])(h))


def _mobile(c):
    L = keras.layers
    x = keras.Input((c["size"], c["size"], c["cin"]))

    def block(t, cout, stride):
        cin = t.shape[-1]
        e = L.ReLU(6.0)(L.BatchNormalization()(L.Conv2D(c["expand"] * cin, 1, padding="same", use_bias=False)(t)))
        e = L.ReLU(6.0)(L.BatchNormalization()(L.DepthwiseConv2D(c["k"], strides=stride, padding="same", use_bias=False)(e)))
        e = L.BatchNormalization()(L.Conv2D(cout, 1, padding="same", use_bias=False)(e))
        return L.Add()([t, e]) if stride == 1 and cin == cout else e

    h = block(block(x, c["cout"], c["stride"]), c["cout"], 1)
    return keras.Model(x, L.Dense(c["classes"])(h))


def _mlp(c):
    L = keras.layers
    x = keras.Input((c["features"],))
    h = L.Dense(c["hidden"], activation="relu")(L.Dense(c["hidden"], activation="relu")(x))
    return keras.Model(x, L.Dense(c["classes"])(h))


def _lstm(c):
    x = keras.Input((c["steps"], c["features"]))
    return keras.Model(x, keras.layers.Dense(c["outputs"])(keras.layers.LSTM(c["units"])(x)))


_BUILD = {"mlp": _mlp, "lm": _decoder, "infer": _decoder, "encode": _encoder, "residual": _residual, "mobile": _mobile, "lstm": _lstm}


# ------------------------------------------------------------------------------------------------ weights and inputs
def _shapes(c):
    """(shape, fan-in) of every trainable weight in the order of ``model.trainable_variables``; fan-in 0: a scale near one, -1: a small vector, -2: the
    shift of a batch normalisation."""
    k, out = c["kind"], []
    if k == "mlp":
        f, h, n = c["features"], c["hidden"], c["classes"]
        return [((f, h), f), ((h,), -1), ((h, h), h), ((h,), -1), ((h, n), h), ((n,), -1)]
    if k == "lstm":
        f, u, o = c["features"], c["units"], c["outputs"]
        return [((f, 4 * u), f), ((u, 4 * u), u), ((4 * u,), -1), ((u, o), u), ((o,), -1)]
    if k in ("lm", "infer", "encode"):
        d, f, n, kv, v = c["d"], c["ffn"], c["heads"], c.get("kv_heads", c["heads"]), c["vocab"]
        hd = d // n
        out.append(((v, d), 4))
        gated = c.get("style") == "gated"
        if k != "encode" and not gated:
            out.append(((c["seq"], d), 16))
        norm = [((d,), 0)] if gated else [((d,), 0), ((d,), -1)]
        for _ in range(c["layers"]):
            if k == "encode":
                for _ in range(3):
                    out += [((d, n, hd), d), ((n, hd), -1)]
                out += [((n, hd, d), d), ((d,), -1)] + norm
                out += [((d, f), d), ((f,), -1), ((f, d), f), ((d,), -1)] + norm
            elif gated:
                out += norm + [((d, n, hd), d), ((d, kv, hd), d), ((d, kv, hd), d), ((n, hd, d), d)] + norm
                out += [((d, f), d), ((d, f), d), ((f, d), f)]
            else:
                out += norm + [((d, n, hd), d)] * 3 + [((n, hd, d), d)] + norm
                out += [((d, f), d), ((f,), -1), ((f, d), f), ((d,), -1)]
        return out if k == "encode" else out + norm + [((d, v), d)]
    bn = lambda ch: [((ch,), 0), ((ch,), -2)]  # noqa: E731
    if k == "residual":
        ci, w, o = c["cin"], c["width"], 4 * c["width"]
        a1, a2, a3 = [((1, 1, ci, w), ci)], [((3, 3, w, w), 9 * w)], [((1, 1, w, o), w)]
        out = a1 + bn(w) + a2 + bn(w) + [((1, 1, ci, o), ci)] + a3 + bn(o) + bn(o)
        out += [((1, 1, o, w), o)] + bn(w) + a2 + bn(w) + a3 + bn(o)
        return out + [((o, c["classes"]), o), ((c["classes"],), -1)]
    for ci in (c["cin"], c["cout"]):
        e, o, kk = c["expand"] * ci, c["cout"], c["k"]
        out += [((1, 1, ci, e), ci)] + bn(e) + [((kk, kk, e, 1), kk * kk)] + bn(e) + [((1, 1, e, o), e)] + bn(o)
    return out + [((c["cout"], c["classes"]), c["cout"]), ((c["classes"],), -1)]


def _generator(seed, stream):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + stream)


def _weights(c, seed):
    # In the convolutional cases the weights are whole 16-bit numbers and the shifts keep most rectifiers open: each rectifier
    # that rounding turns over costs its whole gradient, and the comparison with 64 bits would see little else
    exactly = c["kind"] not in ("residual", "mobile")
    open_at = 1.0 if c["kind"] == "residual" else 1.5  # wider open, and the gradients of the shifts in front of a normalised convolution cancel
    g = _generator(seed, 1)
    out = []
    for shape, fan in _shapes(c):
        t = torch.randn(shape, generator=g, device="cuda")
        t = 1.0 + 0.1 * t if fan == 0 else 0.05 * t if fan == -1 else open_at + 0.5 * t if fan == -2 else t * fan ** -0.5
        out.append(t if exactly else t.bfloat16().float())
    return out


def _inputs(c, seed):
    """(x, y) on the device; ``y`` is ``None`` for inference."""
    g, k, b = _generator(seed, 2), c["kind"], c["batch"]

    def whole(hi, shape, lo=0):
        return torch.randint(lo, hi, shape, generator=g, device="cuda", dtype=torch.int32)

    if k in ("lm", "infer"):
        return whole(c["vocab"], (b, c["seq"])), whole(c["vocab"], (b, c["seq"])) if k == "lm" else None
    if k == "encode":
        x = whole(c["vocab"], (b, c["seq"]), 1)
        lengths = whole(c["seq"] + 1, (b, 1), max(1, c["seq"] // 4))
        return x * (torch.arange(c["seq"], device="cuda") < lengths), None
    if k == "lstm":
        return torch.randn((b, c["steps"], c["features"]), generator=g, device="cuda"), torch.randn((b, c["outputs"]), generator=g, device="cuda")
    if k == "mlp":
        return torch.rand((b, c["features"]), generator=g, device="cuda"), whole(c["classes"], (b,))
    # activations as the layers in front leave them: rectified
    x = torch.randn((b, c["size"], c["size"], c["cin"]), generator=g, device="cuda")
    out = -(-c["size"] // c["stride"])
    return torch.relu(x).bfloat16().float(), whole(c["classes"], (b, out, out))


def prepare(case, seed):
    keras.utils.set_random_seed(int(seed) % 100003)
    float32 = case["kind"] in ("mlp", "lstm")
    keras.config.set_dtype_policy("float32" if float32 else "mixed_bfloat16")
    model = _BUILD[case["kind"]](case)
    weights = _weights(case, seed)
    variables = model.trainable_variables
    assert [tuple(v.shape) for v in variables] == [tuple(w.shape) for w in weights], "weights and model disagree"
    for v, w in zip(variables, weights):
        v.assign(w)
    del weights
    x, y = _inputs(case, seed)
    if y is None:
        real = (x != 0).unsqueeze(-1) if case["kind"] == "encode" else None
        return {"case": case, "model": model, "x": x, "y": None, "real": real}
    if case["kind"] == "lm":
        optimizer = keras.optimizers.AdamW(learning_rate=3e-4, weight_decay=0.1)
    elif float32:
        optimizer = keras.optimizers.Adam(learning_rate=1e-3)
    else:
        optimizer = keras.optimizers.SGD(learning_rate=0.01, momentum=0.9)
    loss = keras.losses.MeanSquaredError() if case["kind"] == "lstm" else keras.losses.SparseCategoricalCrossentropy(from_logits=True)
    model.compile(optimizer=optimizer, loss=loss)
    optimizer.build(model.trainable_variables)
    moments = [v.value for v in optimizer.variables if "momentum" in v.name]
    # Adam divides by the root of the second moment: the first step of a vector that is near zero says little, so of AdamW's
    # weights the matrices are returned (the moments are whole)
    kept = [v for v in model.trainable_variables if case["kind"] != "lm" or len(v.shape) > 1]
    return {"case": case, "model": model, "x": x, "y": y, "moments": moments, "kept": kept}


def run(state):
    model = state["model"]
    if state["y"] is None:
        with torch.no_grad():
            out = model(state["x"], training=False)
            return out if state["real"] is None else out * state["real"]
    loss = model.train_on_batch(state["x"], state["y"])
    return {"loss": float(loss), "moments": state["moments"], "weights": [v.value.detach() for v in state["kept"]]}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _norm(x, w, gated):
    if gated:
        return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + _EPS) * next(w)
    return torch.nn.functional.layer_norm(x, x.shape[-1:], next(w), next(w), _EPS)


def _attend(q, k, v, scale, causal, mask):
    """[B, T, heads, head size] in, head by group to keep the score matrices small."""
    out = torch.empty_like(q) if not q.requires_grad else None
    parts = []
    n, group = q.shape[2], q.shape[2] // k.shape[2]
    t = q.shape[1]
    keep = torch.ones((t, t), dtype=torch.bool, device=q.device).tril() if causal else None
    for i in range(n):
        s = torch.matmul(q[:, :, i], k[:, :, i // group].transpose(1, 2)) * scale
        if keep is not None:
            s = s.masked_fill(~keep, -1e30)
        if mask is not None:
            s = s.masked_fill(~mask, -1e30)
        o = torch.matmul(torch.softmax(s, -1), v[:, :, i // group])
        if out is not None:
            out[:, :, i] = o
        else:
            parts.append(o)
    return out if out is not None else torch.stack(parts, 2)


def _project(x, w, bias=None):
    d = x.shape[-1]
    y = torch.matmul(x, w.reshape(d, -1)).reshape(x.shape[:-1] + tuple(w.shape[1:]))
    return y if bias is None else y + bias


def _exact_decoder(c, w, x):
    w = iter(w)
    gated = c.get("style") == "gated"
    h = torch.nn.functional.embedding(x.long(), next(w))
    if not gated:
        h = h + next(w)
    scale = (c["d"] // c["heads"]) ** -0.5
    for _ in range(c["layers"]):
        a = _norm(h, w, gated)
        q, k, v = (_project(a, next(w)) for _ in range(3))
        h = h + torch.matmul(_attend(q, k, v, scale, True, None).flatten(2), next(w).reshape(c["d"], c["d"]))
        m = _norm(h, w, gated)
        if gated:
            m = torch.nn.functional.silu(torch.matmul(m, next(w))) * torch.matmul(m, next(w))
            h = h + torch.matmul(m, next(w))
        else:
            m = torch.nn.functional.gelu(torch.matmul(m, next(w)) + next(w))
            h = h + torch.matmul(m, next(w)) + next(w)
    h = _norm(h, w, gated)
    return torch.matmul(h, next(w))


def _exact_encoder(c, w, x):
    w = iter(w)
    h = torch.nn.functional.embedding(x.long(), next(w))
    real = x != 0
    mask = real[:, :, None] & real[:, None, :]
    scale = (c["d"] // c["heads"]) ** -0.5
    for _ in range(c["layers"]):
        q, k, v = (_project(h, next(w), next(w)) for _ in range(3))
        a = torch.matmul(_attend(q, k, v, scale, False, mask).flatten(2), next(w).reshape(c["d"], c["d"])) + next(w)
        h = _norm(h + a, w, False)
        m = torch.nn.functional.gelu(torch.matmul(h, next(w)) + next(w))
        m = torch.matmul(m, next(w)) + next(w)
        h = _norm(h + m, w, False)
    return h * real[:, :, None]


def _conv64(x, w, stride, groups=1):
    k, size = w.shape[0], x.shape[-1]
    out = -(-size // stride)
    total = max((out - 1) * stride + k - size, 0)
    x = torch.nn.functional.pad(x, (total // 2, total - total // 2, total // 2, total - total // 2))
    if w.shape[0] == 1:
        return torch.einsum("nchw,co->nohw", x[:, :, ::stride, ::stride], w[0, 0])
    if groups > 1:  # tap by tap: no library has a quick depthwise convolution in 64 bits
        y = 0
        for r in range(k):
            for s in range(k):
                y = y + x[:, :, r:r + (out - 1) * stride + 1:stride, s:s + (out - 1) * stride + 1:stride] * w[r, s, :, 0].view(1, -1, 1, 1)
        return y
    y = 0
    for r in range(k):
        for s in range(k):
            y = y + torch.einsum("nchw,co->nohw", x[:, :, r:r + (out - 1) * stride + 1:stride, s:s + (out - 1) * stride + 1:stride], w[r, s])
    return y


def _bn64(x, g, b, eps):
    return torch.nn.functional.batch_norm(x, None, None, g, b, True, 0.0, eps)


def _exact_residual(c, w, x):
    w = list(w)
    x = x.permute(0, 3, 1, 2)
    s = c["stride"]
    eps, relu = 1.001e-5, torch.relu
    t = relu(_bn64(_conv64(x, w[0], s), w[1], w[2], eps))
    t = relu(_bn64(_conv64(t, w[3], 1), w[4], w[5], eps))
    short, t = _conv64(x, w[6], s), _conv64(t, w[7], 1)
    h = relu(_bn64(short, w[8], w[9], eps) + _bn64(t, w[10], w[11], eps))
    t = relu(_bn64(_conv64(h, w[12], 1), w[13], w[14], eps))
    t = relu(_bn64(_conv64(t, w[15], 1), w[16], w[17], eps))
    h = relu(h + _bn64(_conv64(t, w[18], 1), w[19], w[20], eps))
    return torch.matmul(h.permute(0, 2, 3, 1), w[21]) + w[22]


def _exact_mobile(c, w, x):
    w = iter(w)
    h = x.permute(0, 3, 1, 2)
    for cin, stride in ((c["cin"], c["stride"]), (c["cout"], 1)):
        e = _bn64(_conv64(h, next(w), 1), next(w), next(w), 1e-3).clamp(0, 6)
        e = _bn64(_conv64(e, next(w), stride, c["expand"] * cin), next(w), next(w), 1e-3).clamp(0, 6)
        e = _bn64(_conv64(e, next(w), 1), next(w), next(w), 1e-3)
        h = h + e if stride == 1 and cin == c["cout"] else e
    return torch.matmul(h.permute(0, 2, 3, 1), next(w)) + next(w)


def _exact_mlp(c, w, x):
    h = torch.relu(torch.matmul(x, w[0]) + w[1])
    h = torch.relu(torch.matmul(h, w[2]) + w[3])
    return torch.matmul(h, w[4]) + w[5]


def _exact_lstm(c, w, x):
    u = c["units"]
    h = c_ = torch.zeros((x.shape[0], u), dtype=x.dtype, device=x.device)
    z = torch.matmul(x, w[0]) + w[2]
    for t in range(x.shape[1]):
        i, f, g, o = (z[:, t] + torch.matmul(h, w[1])).split(u, -1)
        c_ = torch.sigmoid(f) * c_ + torch.sigmoid(i) * torch.tanh(g)
        h = torch.sigmoid(o) * torch.tanh(c_)
    return torch.matmul(h, w[3]) + w[4]


_EXACT = {"mlp": _exact_mlp, "lm": _exact_decoder, "infer": _exact_decoder, "encode": _exact_encoder, "residual": _exact_residual, "mobile": _exact_mobile,
          "lstm": _exact_lstm}


def exact(case, seed):
    k = case["kind"]
    x, y = _inputs(case, seed)
    w = [t.double() for t in _weights(case, seed)]
    x = x.double() if x.is_floating_point() else x
    if y is None:
        with torch.no_grad():
            return _EXACT[k](case, w, x)
    for t in w:
        t.requires_grad_(True)
    out = _EXACT[k](case, w, x)
    if k == "lstm":
        loss = torch.mean((out - y.double()) ** 2)
    else:
        loss = torch.nn.functional.cross_entropy(out.reshape(-1, out.shape[-1]), y.reshape(-1).long())
    grads = torch.autograd.grad(loss, w)
    moments, weights = [], []
    for t, g in zip(w, grads):
        t = t.detach()
        if k in ("residual", "mobile"):
            m = -0.01 * g
            new = t + m
        else:
            lr = 3e-4 if k == "lm" else 1e-3
            m, v = 0.1 * g, 0.001 * g * g
            new = t * (1 - lr * 0.1) if k == "lm" else t
            new = new - lr * math.sqrt(1 - 0.999) / (1 - 0.9) * m / (torch.sqrt(v) + 1e-7)
        moments.append(m)
        if k != "lm" or t.ndim > 1:
            weights.append(new)
    return {"loss": float(loss.detach()), "moments": moments, "weights": weights}


# ------------------------------------------------------------------------------------------------ work and precision
def work(case):
    k, b = case["kind"], case["batch"]
    params = sum(math.prod(s) for s, _ in _shapes(case))
    training = k not in ("infer", "encode")
    # weights are read once; a training step reads and writes them and the optimizer's moments
    slots = {"lm": 2, "mlp": 2, "lstm": 2, "residual": 1, "mobile": 1}.get(k, 0)
    size = params * 4 * (2 + 2 * slots) if training else params * 2
    if k == "mlp":
        macs = b * (case["features"] * case["hidden"] + case["hidden"] ** 2 + case["hidden"] * case["classes"])
        size += 4 * b * case["features"]
    elif k == "lstm":
        macs = b * case["steps"] * 4 * case["units"] * (case["features"] + case["units"])
        size += 4 * b * case["steps"] * (case["features"] + 2 * 5 * case["units"])  # the state of each step, kept for the way back
    elif k in ("lm", "infer", "encode"):
        d, t, tokens = case["d"], case["seq"], b * case["seq"]
        kv = case.get("kv_heads", case["heads"]) * d // case["heads"]
        layer = 2 * d * d + 2 * d * kv + (3 if case.get("style") == "gated" else 2) * d * case["ffn"]
        attention = 2 * t * d * (1.0 if k == "encode" else 0.5)
        macs = tokens * case["layers"] * (layer + attention) + (0 if k == "encode" else tokens * d * case["vocab"])
        if k == "lm":
            # the inputs of the products and of the norms and the logits, kept for the way back
            size += 2 * tokens * (2 * case["layers"] * (8 * d + 2 * case["ffn"]) + 4 * case["vocab"])
        else:
            size += 2 * tokens * (d if k == "encode" else case["vocab"])
    else:
        s, n, o, stride = case["size"], 0, -(-case["size"] // case["stride"]), case["stride"]
        if k == "residual":
            ci, w = case["cin"], case["width"]
            convs = [(o, ci, w, 1), (o, w, w, 9), (o, w, 4 * w, 1), (o, ci, 4 * w, 1), (o, 4 * w, w, 1), (o, w, w, 9), (o, w, 4 * w, 1)]
        else:
            convs = []
            for ci, si, so in ((case["cin"], s, o), (case["cout"], o, o)):
                e = case["expand"] * ci
                convs += [(si, ci, e, 1), (so, 1, e, case["k"] ** 2), (so, e, case["cout"], 1)]
        macs = sum(b * so * so * ci * co * taps for so, ci, co, taps in convs) + b * o * o * convs[-1][2] * case["classes"]
        size += 4 * b * s * s * case["cin"]
        # each activation written, normalised and read on the way there, and its gradient twice on the way back, in 16 bits
        size += sum(2 * b * so * so * co * 5 for so, _, co, _ in convs)
    return {"bytes": int(size), "flops": int(2 * macs * (3 if training else 1))}


def tolerance(case):
    # about four times the largest error against 64 bits over listed and drawn cases: 5e-7 in float32, 0.007 of logits and
    # states, 0.01 of a decoder's gradients; a convolutional step's first gradients are 0.02 to 0.04 off, because each rectifier
    # that rounding turns over adds its whole gradient: two implementations round most of them alike
    return {"rel": {"mlp": 1e-5, "lstm": 1e-5}.get(case["kind"], 0.03)}
