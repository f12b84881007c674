"""Kernels and dispatch rules at the sizes where they change over, against plain PyTorch in 64 bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


# ------------------------------------------------------------------------------------------------ LSTM on clusters
# every height of a row tile (2, 4, 8, 10 rows) with its remainders, every K width (64, 128, 192, 256 units), units that end inside a CTA's
# sixteen, several tiles a cluster (300 rows), more clusters than run at once (2500 rows), the first size beyond the clusters (260)
@pytest.mark.parametrize("B,T,U", [(1, 1, 4), (7, 2, 256), (28, 3, 256), (50, 3, 248), (64, 12, 256), (71, 3, 256), (300, 3, 256), (2500, 2, 24), (33, 3, 128),
                                   (40, 6, 176), (64, 4, 48), (5, 6, 68), (9, 3, 260), (85, 3, 252), (512, 2, 176), (768, 2, 192), (1024, 2, 96), (403, 2, 256)])
@pytest.mark.parametrize("reverse,sequence,states", [(False, True, True), (True, False, False)])
def test_lstm_on_clusters_against_the_steps_in_64_bits(B, T, U, reverse, sequence, states):
    from keras_b200.kernels import gemm, lstm

    g = torch.Generator(device="cuda").manual_seed(B + U)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    args = [rnd(B, T, 4 * U), rnd(4 * U), 0.5 * rnd(B, U), rnd(B, U), rnd(U, 4 * U) * U ** -0.5]
    wanted = [True, True, states, states, True]
    mine = [a.clone().requires_grad_(n) for a, n in zip(args, wanted)]
    exact = [a.double().requires_grad_(n) for a, n in zip(args, wanted)]
    results, want = lstm.run(*mine, reverse, sequence), lstm._composed(*exact, reverse)
    up = [rnd(B, T, U), rnd(B, U), rnd(B, U)]
    pairs = [(r, w, u) for r, w, u in zip(results, want, up) if r is not None]
    sum((r * u).sum() for r, _, u in pairs).backward()
    sum((w * u).sum() for _, w, u in pairs).backward()
    gemm.check_errors()
    for r, w, _ in pairs:
        assert _rel(r, w) < 3e-6  # fp32 sums over U terms a step, a few steps deep
    for a, b, n in zip(mine, exact, wanted):
        assert not n or _rel(a.grad, b.grad) < 1e-5  # up to B * T terms in the weight gradient


# ------------------------------------------------------------------------------------------------ products of odd width
# the last width in multiples of 8, the first and the fullest in multiples of 64, one that is a multiple of 8
@pytest.mark.parametrize("N,pitch", [(1023, 1024), (1025, 1088), (1087, 1088), (1032, 1032), (8009, 8064)])
def test_odd_widths_are_computed_in_whole_lines(N, pitch):
    from keras_b200.kernels import gemm
    from keras_b200.kernels import ops as kops

    g = torch.Generator(device="cuda").manual_seed(N)
    M, K = 300, 128
    x = torch.randn((M, K), generator=g, device="cuda").bfloat16().requires_grad_(True)
    w = (torch.randn((K, N), generator=g, device="cuda") * K ** -0.5).bfloat16().requires_grad_(True)
    b = torch.randn(N, generator=g, device="cuda").requires_grad_(True)
    labels = torch.randint(0, N, (M,), generator=g, device="cuda")
    y = gemm.GemmFn.apply(x, w, b)
    assert gemm.padded_width(N) == pitch and y.shape == (M, N) and y.stride() == (pitch, 1)
    seen = []
    y.register_hook(seen.append)
    kops.FusedSoftmaxXent.apply(y, labels).sum().backward()
    gemm.check_errors()
    assert seen[0].stride() == (pitch, 1) and not seen[0].as_strided((M, pitch), (pitch, 1))[:, N:].any()
    exact = [t.detach().double().requires_grad_(True) for t in (x, w, b)]
    want = exact[0] @ exact[1] + exact[2]
    torch.nn.functional.cross_entropy(want, labels, reduction="sum").backward()
    # logits rounded to bf16 (2^-9 of values up to 5), and their gradient with them
    assert _rel(y.detach(), want.detach()) < 2.0 ** -8
    for got, ref in zip((x, w, b), exact):
        assert _rel(got.grad, ref.grad) < 2.0 ** -6


# ------------------------------------------------------------------------------------------------ weight gradients over many rows
# the edges of a tile (32, 64 rows, 128 columns) and of a block of K (16), one slice and many, rows that are copied value by value
@pytest.mark.parametrize("K,M,N", [(1, 1, 1), (15, 3, 5), (16, 32, 128), (17, 33, 129), (33, 31, 127), (200, 64, 256), (1030, 65, 132), (3000, 250, 1000), (6400, 256, 1024),
                                   (40000, 8, 48)])
@pytest.mark.parametrize("kept", [False, True])
def test_weight_gradient_of_many_rows(K, M, N, kept):
    from keras_b200.kernels import sgemm, shadow

    g = torch.Generator(device="cuda").manual_seed(K + M)
    a = torch.randn((K, M + 4), generator=g, device="cuda")[:, :M]  # a row pitch of its own
    b = torch.randn((K, N), generator=g, device="cuda")
    if kept:
        targets = [torch.nn.Parameter(torch.zeros(s, device="cuda")) for s in ((M, N), (N,))]
        for t in targets:
            t.grad = torch.ones_like(t)
        with shadow.arena_backward():
            assert sgemm.weight_gradient(a, b, *targets, sums=True) == (None, None)
        w, s = (t.grad for t in targets)
    else:
        w, s = sgemm.weight_gradient(a, b, sums=True)
        assert torch.equal(w, sgemm.weight_gradient(a, b)[0])
    # any order of K products and sums errs by K + 2 roundings of 2^-24 of the sum of magnitudes at most
    bound, old = (K + 2) * 2.0 ** -24, 1.0 if kept else 0.0
    assert ((w.double() - old - a.double().t() @ b.double()).abs() <= bound * (a.double().abs().t() @ b.double().abs() + old)).all()
    assert ((s.double() - old - b.double().sum(0)).abs() <= bound * (b.double().abs().sum(0) + old)).all()


@pytest.mark.parametrize("F,bias", [(4, True), (24, True), (24, False)])  # the library's product, this package's
def test_lstm_layer_weight_gradients_in_place_and_twice(F, bias):
    import keras_b200 as keras
    from keras_b200.kernels import lstm, shadow

    keras.utils.set_random_seed(0)
    layer = keras.layers.LSTM(20, return_sequences=True, use_bias=bias)
    x = torch.randn(128, 9, F, device="cuda")
    up = torch.randn(128, 9, 20, device="cuda")
    layer(x)
    weights = [v._value for v in layer.trainable_variables]
    exact = [w.detach().double().requires_grad_(True) for w in weights]
    zero = torch.zeros(128, 20, device="cuda", dtype=torch.float64)
    want = torch.autograd.grad((lstm._composed(x.double() @ exact[0], exact[2] if bias else None, zero, zero, exact[1], False)[0] * up).sum(), exact)
    grads = torch.autograd.grad((layer(x) * up).sum(), weights)
    for w in weights:
        w.grad = torch.zeros_like(w)
    with shadow.arena_backward():
        (layer(x) * up).sum().backward()
    for w, mine, ref in zip(weights, grads, want):
        assert _rel(mine, ref) < 1e-5 and _rel(w.grad, ref) < 1e-5  # up to 1152 terms each
        w.grad = None
    twice = torch.autograd.grad((layer(x) * up).sum(), weights, create_graph=True)
    for mine, ref in zip(twice, want):
        assert _rel(mine.detach(), ref) < 1e-5
    assert all(torch.isfinite(t).all() for t in torch.autograd.grad(sum((t ** 2).sum() for t in twice), weights))


# ------------------------------------------------------------------------------------------------ products of inference
@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("M,K,widths", [(1, 64, (64,)), (7, 72, (72,)), (77, 768, (1001,)), (128, 200, (264,)), (128, 3072, (64, 64, 128)), (33, 256, (1024, 256, 256)),
                                        (129, 64, (64,)), (300, 200, (1001,)), (257, 768, (192, 64, 64)), (130, 512, (4099,))])
def test_inference_products_read_weights_as_stored(M, K, widths, fp32):
    """Few rows straight from the weight, more through one bf16 matrix; any width, one weight or three, every epilogue."""
    from keras_b200.kernels import gemm
    from keras_b200.models import direct

    g = torch.Generator(device="cuda").manual_seed(M + K)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    ws = [torch.randn(K, n, generator=g, device="cuda") * K ** -0.5 for n in widths]
    bs = [torch.randn(n, generator=g, device="cuda") for n in widths]
    ws = ws if fp32 else [w.bfloat16() for w in ws]
    acts = {0: lambda t: t, 1: torch.relu, 3: torch.nn.functional.silu, 4: torch.nn.functional.gelu}
    for act, fn in acts.items():
        for biases in ([None] * len(ws), bs, [b.bfloat16() for b in bs]):
            out = direct._product(x, ws, biases, act)
            ref = torch.cat([x.double() @ w.bfloat16().double() + (0 if b is None else b.double()) for w, b in zip(ws, biases)], 1)
            # exact products of bf16, summed in fp32, one rounding to bf16
            assert _rel(out[:, :sum(widths)], fn(ref)) < 2.0 ** -8
            if biases[0] is None:
                assert not out[:, sum(widths):].float().any()
            assert torch.equal(out, direct._product(x, ws, biases, act))
    gemm.check_errors()


def _models(keras):
    L = keras.layers

    def tokens(layer):
        i = keras.Input((24,), dtype="int32")
        return keras.Model(i, layer(i))

    def decoder(i):
        h = L.Embedding(301, 128)(i)
        a = L.MultiHeadAttention(2, 64, use_bias=True)(L.LayerNormalization()(h), L.LayerNormalization()(h))
        h = L.Add()([h, a])
        n = L.LayerNormalization()(h)
        n = L.MultiHeadAttention(2, 64, use_bias=False)(n, n, use_causal_mask=True)
        h = L.Add()([h, n])
        m = L.LayerNormalization(center=False)(h)
        h = L.Add()([h, L.Dense(128)(L.Dense(256, activation="gelu")(m))])
        return L.Dense(301)(L.LayerNormalization()(h))

    def gated(i):
        h = L.Embedding(301, 256)(i)
        a = L.RMSNormalization()(h)
        h = L.Add()([h, L.GroupedQueryAttention(64, 4, 2, use_bias=False)(a, a, use_causal_mask=True)])
        m = L.RMSNormalization()(h)
        m = L.Multiply()([L.Dense(512, activation="silu")(m), L.Dense(512, activation=lambda t: t * 2)(m)])
        return L.Add()([h, L.Dense(256)(m)])

    def padded(i):
        h = L.Embedding(301, 128, mask_zero=True)(i)
        for _ in range(2):
            h = L.LayerNormalization()(L.Add()([h, L.MultiHeadAttention(2, 64)(h, h)]))
            h = L.LayerNormalization()(L.Add()([h, L.Dense(128, activation="relu")(h)]))
        return h

    return {"decoder": tokens(decoder), "gated": tokens(gated), "padded": tokens(padded)}


@pytest.mark.parametrize("policy", ["mixed_bfloat16", "bfloat16"])
@pytest.mark.parametrize("batch", [1, 2, 40])
def test_layers_called_directly_agree_with_their_own_calls(policy, batch, monkeypatch):
    import keras_b200 as keras
    from keras_b200.models import direct

    keras.utils.set_random_seed(3)
    keras.config.set_dtype_policy(policy)
    try:
        models = _models(keras)
    finally:
        keras.config.set_dtype_policy("float32")
    ids = torch.randint(-1, 301, (batch, 24), device="cuda", dtype=torch.int32)
    ids[:, 17:] = 0
    for name, model in models.items():
        with torch.no_grad():
            model(ids)  # the first call is the layers' own
            taken = []
            for fn in ("_dense", "_attention", "add_norm", "_embedding"):
                plain = getattr(direct, fn)
                monkeypatch.setattr(direct, fn, lambda *a, _f=plain, _n=fn: (lambda r: (taken.append(_n) if r is not None else None, r)[1])(_f(*a)))
            direct._PLANS.clear()
            mine = model(ids)
            monkeypatch.undo()
            direct._PLANS.clear()
            assert {"_dense", "_attention", "add_norm", "_embedding"} <= set(taken), (name, taken)
            monkeypatch.setattr(direct, "usable", lambda x: False)
            own = model(ids)
            monkeypatch.undo()
        assert mine.shape == own.shape and mine.dtype == own.dtype
        # bf16 throughout, some ten roundings deep; bit for bit below
        assert _rel(mine.float(), own.double()) < 0.02, name
        a, b = getattr(mine, "_keras_mask", None), getattr(own, "_keras_mask", None)
        assert (a is None) == (b is None) and (a is None or torch.equal(a, b))


@pytest.mark.parametrize("policy", ["mixed_bfloat16", "bfloat16"])
@pytest.mark.parametrize("batch", [1, 2, 5, 40])
def test_a_second_call_repeats_the_first_bit_for_bit(policy, batch):
    """The first call of a model is its layers' own, the next are made directly."""
    import keras_b200 as keras

    keras.utils.set_random_seed(3)
    keras.config.set_dtype_policy(policy)
    try:
        models = _models(keras)
    finally:
        keras.config.set_dtype_policy("float32")
    g = torch.Generator(device="cuda").manual_seed(batch)
    ids = torch.randint(0, 301, (batch, 24), device="cuda", dtype=torch.int32, generator=g)
    for name, model in models.items():
        for v in model.trainable_variables:
            v.assign(v.value.float() + 0.3 * torch.randn(tuple(v.shape), device="cuda", generator=g))
        with torch.no_grad():
            assert torch.equal(model(ids), model(ids)), name


@pytest.mark.parametrize("policy", ["mixed_bfloat16", "bfloat16"])
@pytest.mark.parametrize("M,K,N", [(1, 768, 768), (77, 768, 3072), (77, 3072, 768), (64, 512, 1024), (13, 64, 64), (128, 264, 15000), (7, 72, 14336), (77, 64, 14337),
                                   (8, 128, 304), (200, 64, 64), (300, 256, 1001), (130, 2048, 520)])
@pytest.mark.parametrize("activation,bias", [(None, False), (None, True), ("relu", True), ("gelu", True), ("silu", False), ("silu", True)])
def test_dense_called_directly_has_the_bits_of_its_own_call(policy, M, K, N, activation, bias):
    """Both sides of every rule: the library's products and this package's, few rows and many, wide and narrow."""
    import keras_b200 as keras
    from keras_b200.models import direct

    layer = keras.layers.Dense(N, activation=activation, use_bias=bias, dtype=policy)
    layer.build((None, K))
    if bias:
        layer.bias.assign(torch.randn(N, device="cuda"))
    x = torch.randn(M, K, device="cuda").bfloat16()
    with torch.no_grad():
        own = layer(x)
        taken = direct._dense(layer, x)
    assert taken is not None and torch.equal(own, taken)


def test_direct_calls_at_every_new_batch(monkeypatch):
    """Sizes that alternate, and one that is new, are called directly throughout; a wrong one raises what the layer's own call raises."""
    import keras_b200 as keras
    from keras_b200.models import direct

    keras.config.set_dtype_policy("mixed_bfloat16")
    try:
        i = keras.Input((None, 64))
        model = keras.Model(i, keras.layers.Dense(96)(keras.layers.LayerNormalization()(keras.layers.Dense(128, activation="gelu")(i))))
        narrow = keras.layers.Dense(64)
        narrow(torch.zeros(2, 32, device="cuda"))
    finally:
        keras.config.set_dtype_policy("float32")
    taken, plain = [], direct._dense

    def counted(layer, x):
        out = plain(layer, x)
        taken.append(out is not None)
        return out

    monkeypatch.setattr(direct, "_dense", counted)
    with torch.no_grad():
        model(torch.randn(2, 5, 64, device="cuda"))
        for b, t in ((2, 5), (3, 7), (2, 5), (3, 7), (200, 9)):
            x = torch.randn(b, t, 64, device="cuda")
            del taken[:]
            mine = model(x)
            assert taken == [True, True], (b, t)
            with monkeypatch.context() as m:
                m.setattr(direct, "usable", lambda x: False)
                assert torch.equal(mine, model(x))
        assert plain(narrow, torch.randn(2, 64, device="cuda").bfloat16()) is None
    with pytest.raises(ValueError, match="incompatible"):
        narrow(torch.zeros(2, 64, device="cuda"))


def test_direct_calls_see_every_change_of_a_layer(monkeypatch):
    import keras_b200 as keras
    from keras_b200.models import direct

    keras.utils.set_random_seed(4)
    keras.config.set_dtype_policy("mixed_bfloat16")
    try:
        i = keras.Input((128,))
        first, second = keras.layers.Dense(128, activation="relu"), keras.layers.Dense(64)
        model = keras.Model(i, second(first(i)))
    finally:
        keras.config.set_dtype_policy("float32")
    x = torch.randn(9, 128, device="cuda")

    def both():
        with torch.no_grad():
            model(x)
            mine = model(x)
            monkeypatch.setattr(direct, "usable", lambda x: False)
            own = model(x)
            monkeypatch.undo()
        assert _rel(mine.float(), own.double()) < 0.01 or not own.any()
        return mine

    seen = [both()]
    first.activation = keras.activations.silu
    seen.append(both())
    first.activation = lambda t: t + 1
    seen.append(both())
    first.kernel.assign(first.kernel * 0.5)
    seen.append(both())
    first.kernel.value.data.mul_(2.0)  # past the version counter
    seen.append(both())
    first.call = lambda inputs, training=None: inputs * 0
    seen.append(both())
    del first.call
    second.enable_lora(4)
    second.lora_kernel_b.assign(torch.randn(4, 64, device="cuda"))
    seen.append(both())
    second.quantize("int8")
    seen.append(both())
    assert all(not torch.equal(a, b) for a, b in zip(seen, seen[1:]))
    trained = keras.Model(i, first(i))
    trained.compile(keras.optimizers.SGD(0.5), "mse")
    trained.train_on_batch(x, torch.zeros(9, 128, device="cuda"))  # weights now have 16-bit shadows
    with torch.no_grad():
        mine = trained(x)
        ref = torch.matmul(x.bfloat16().double(), first._kernel._value.bfloat16().double()) + first.bias._value.double() + 1
    assert _rel(mine.float(), ref) < 0.01


# ------------------------------------------------------------------------------------------------ residual sums with their normalisation
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,D", [(1, 8), (50, 100), (5, 200), (700, 256), (2664, 512), (1500, 768), (33, 776), (900, 1024), (77, 2048), (40, 4096), (9, 8192)])
@pytest.mark.parametrize("rms", [False, True])
def test_add_and_norm_in_one_pass(rows, D, dtype, rms):
    from keras_b200.kernels import ops as kops

    g = torch.Generator(device="cuda").manual_seed(D)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    mine = [rnd(rows, D).to(dtype).requires_grad_(True), rnd(rows, D).to(dtype).requires_grad_(True), rnd(D).requires_grad_(True)]
    mine.append(None if rms else rnd(D).requires_grad_(True))
    up = (rnd(rows, D).to(dtype), rnd(rows, D).to(dtype))
    total, y = kops.FusedAddNorm.apply(*mine, 1e-5, rms)
    exact = [None if t is None else t.detach().double().requires_grad_(True) for t in mine]
    s = exact[0] + exact[1]
    s = s + (s.to(dtype).double() - s).detach()  # the sum is rounded to its type before it is normalised
    n = torch.nn.functional.rms_norm(s, (D,), exact[2], 1e-5) if rms else torch.nn.functional.layer_norm(s, (D,), exact[2], exact[3], 1e-5)
    assert torch.equal(total, mine[0] + mine[1])
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-6  # one rounding of each result; fp32 sums of at most 8192 values
    assert _rel(y, n) < tol
    for outs in ((0, 1), (1,), (0,)):  # either result may have no gradient
        have = [t for t in mine if t is not None]
        a = torch.autograd.grad([(total, y)[k] for k in outs], have, [up[k] for k in outs], retain_graph=True, allow_unused=True)
        b = torch.autograd.grad([(s, n)[k] for k in outs], [t for t in exact if t is not None], [up[k].double() for k in outs], retain_graph=True, allow_unused=True)
        for p, q in zip(a, b):
            assert (p is None) == (q is None) and (p is None or _rel(p, q) < (tol if p.ndim > 1 else 1e-4 if dtype == torch.bfloat16 else 1e-5))


def test_add_and_norm_second_derivatives():
    from keras_b200.kernels import ops as kops

    a, b = (torch.randn(6, 64, device="cuda", requires_grad=True) for _ in range(2))
    gamma, beta = (torch.randn(64, device="cuda", requires_grad=True) for _ in range(2))
    second = []
    for f in (lambda: kops.FusedAddNorm.apply(a, b, gamma, beta, 1e-5, False),
              lambda: (a + b, torch.nn.functional.layer_norm(a + b, (64,), gamma, beta, 1e-5))):
        t, y = f()
        (g,) = torch.autograd.grad((y ** 2).sum() + (t ** 3).sum(), a, create_graph=True)
        second.append(torch.autograd.grad((g ** 2).sum(), [a, b, gamma]))
    for p, q in zip(*second):
        assert torch.allclose(p, q, rtol=1e-4, atol=1e-4 * q.abs().max().item())


# ------------------------------------------------------------------------------------------------ several products in one launch
@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("M,K,widths", [(128, 64, (64, 64, 64)), (333, 192, (128, 64, 64)), (2664, 512, (512, 512, 512)), (300, 256, (1024, 256, 256)), (200, 64, (320, 72))])
def test_grouped_products(variant, M, K, widths):
    from keras_b200.kernels import gemm
    from keras_b200.kernels import ops as kops

    g = torch.Generator(device="cuda").manual_seed(M)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, ws, dys = rnd(M, K), [rnd(K, n) for n in widths], [rnd(M, n) for n in widths]
    bs = [torch.randn(n, generator=g, device="cuda") for n in widths]
    real = kops._lib().kb200_gemm_group
    plain, kops._lib().kb200_gemm_group = real, lambda *a: real(*a[:11], kops._i(variant), *a[12:])  # this kernel, whatever the rule says
    try:
        for biases in ([None] * len(ws), bs, [b.bfloat16() for b in bs]):
            outs = [torch.empty(M, n, device="cuda", dtype=torch.bfloat16) for n in widths]
            gemm.group([(x, w, o, b) for w, o, b in zip(ws, outs, biases)], M, 0, 1, False)
            for w, o, b in zip(ws, outs, biases):
                assert _rel(o, x.double() @ w.double() + (0 if b is None else b.double())) < 2.0 ** -8
        for split in (1, 2):
            if variant == 1 and split > 1:
                continue
            grads = [torch.full((K, n), 3.0, device="cuda") for n in widths]
            gemm.group([(x, dy, d, None) for dy, d in zip(dys, grads)], K, 1, 1, False, split_k=split, accumulate=True)
            for dy, d in zip(dys, grads):
                assert _rel(d, 3.0 + x.double().t() @ dy.double()) < 2.0 ** -17
        if all(n % 64 == 0 for n in widths):
            dx = torch.empty(M, K, device="cuda", dtype=torch.bfloat16)
            gemm.group([(dy, w, dx, None) for dy, w in zip(dys, ws)], M, 0, 0, True)
            assert _rel(dx, sum(dy.double() @ w.double().t() for dy, w in zip(dys, ws))) < 2.0 ** -8
    finally:
        kops._lib().kb200_gemm_group = plain
    gemm.check_errors()


@pytest.mark.parametrize("grouped,bias", [(False, False), (False, True), (True, True)])
def test_attention_layers_take_their_projections_together(grouped, bias, monkeypatch):
    """The same outputs and gradients as three layers of their own, inside and outside an arena's backward pass."""
    import keras_b200 as keras
    from keras_b200.kernels import gemm

    def step(joint):
        keras.utils.set_random_seed(5)
        keras.config.set_dtype_policy("mixed_bfloat16")
        try:
            i = keras.Input((96, 256))
            layer = keras.layers.GroupedQueryAttention(64, 4, 2, use_bias=bias) if grouped else keras.layers.MultiHeadAttention(4, 64, use_bias=bias)
            h = keras.layers.LayerNormalization()(keras.layers.Dense(256)(i))
            model = keras.Model(i, keras.layers.Dense(8)(layer(h, h, use_causal_mask=True)))
        finally:
            keras.config.set_dtype_policy("float32")
        if not joint:
            monkeypatch.setattr(gemm, "projections", lambda *a: None)
        used = []
        plain = gemm.ProjectionsFn.apply
        monkeypatch.setattr(gemm.ProjectionsFn, "apply", lambda *a: (used.append(1), plain(*a))[1])
        x = torch.randn(4, 96, 256, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1), requires_grad=True)
        model(x)
        y = model(x)
        grads = torch.autograd.grad((y.float() ** 2).sum(), [x] + [v.value for v in model.trainable_variables])
        model.compile(keras.optimizers.SGD(0.1, momentum=0.9), "mse")
        for _ in range(3):
            model.train_on_batch(x.detach(), torch.zeros(4, 96, 8, device="cuda"))
        monkeypatch.undo()
        assert bool(used) == joint
        return [y, *grads, *[v.value.detach().clone() for v in model.trainable_variables]]

    for a, b in zip(step(True), step(False)):
        # bf16 gradients; the input's is rounded once instead of three times.  A key's bias has none: what is there is rounding
        assert _rel(a.float(), b.double()) < 0.02 or b.abs().max() < 1e-5
    gemm.check_errors()


# ------------------------------------------------------------------------------------------------ cross-entropy with its gradient
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,V,ld", [(3, 2049, 2056), (130, 5001, 5008), (65, 8009, 8016), (64, 50257, 50264)])
def test_cross_entropy_that_makes_its_gradient_ahead(rows, V, ld, dtype):
    from keras_b200.kernels import ops as kops

    buf = (torch.randn(rows, ld, device="cuda") * 3).to(dtype)
    buf[:, 3:17] = float("-inf")
    labels = torch.randint(20, V, (rows,), device="cuda")
    labels[1] = -1
    expected = torch.full((rows,), 1.0 / rows, device="cuda")
    other = expected.clone()
    other[::3] *= 2
    other[2] = float("nan")
    results = []
    for ahead in (True, False):
        for upstream in (expected, other, torch.zeros_like(expected)):
            logits = buf.clone()[:, :V].requires_grad_(True)
            with kops.gradient_follows():
                if ahead:
                    kops.expect_upstream(lambda n: 1.0 / n)
                loss = kops.FusedSoftmaxXent.apply(logits, labels)
            first = torch.autograd.grad(loss, logits, upstream, retain_graph=True)[0].clone()
            again = torch.autograd.grad(loss, logits, upstream)[0]  # a second pass has no gradient made ahead
            assert torch.equal(first, again) or upstream is other and torch.equal(first.nan_to_num(), again.nan_to_num())
            results.append((loss.detach(), first.nan_to_num()))
    for (la, ga), (lb, gb) in zip(results[:3], results[3:]):
        assert torch.equal(la, lb) and torch.equal(ga, gb)


# ------------------------------------------------------------------------------------------------ float32 products of few rows
@pytest.mark.parametrize("M,K,N", [(1, 16, 1), (16, 17, 64), (77, 130, 33), (128, 784, 512), (128, 512, 10), (256, 500, 1000), (64, 64, 64), (65, 2048, 65)])
@pytest.mark.parametrize("relu,bias", [(True, True), (False, False), (False, True)])
def test_float32_dense_products(M, K, N, relu, bias):
    from keras_b200.kernels import sgemm

    g = torch.Generator(device="cuda").manual_seed(M)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    mine = [rnd(M, K).requires_grad_(True), (rnd(K, N) * K ** -0.5).requires_grad_(True)] + ([rnd(N).requires_grad_(True)] if bias else [])
    out = sgemm.DenseFn.apply(mine[0], mine[1], mine[2] if bias else None, None, None, relu)
    exact = [t.detach().double().requires_grad_(True) for t in mine]
    ref = exact[0] @ exact[1] + (exact[2] if bias else 0)
    ref = ref * (out.detach() > 0) if relu else ref  # the rectifier as the fp32 sum decides it
    up = rnd(M, N)
    assert _rel(out, ref) < 2e-6 or not ref.any()  # fp32 products, sums of at most 2048 of them
    for a, b in zip(torch.autograd.grad(out, mine, up), torch.autograd.grad(ref, exact, up.double())):
        assert _rel(a, b) < 2e-6 or not b.any()


def test_float32_dense_layer_keeps_nan_and_second_derivatives():
    import keras_b200 as keras

    layer = keras.layers.Dense(32, activation="relu")
    x = torch.randn(8, 48, device="cuda", requires_grad=True)
    y = layer(x)
    assert "DenseFn" in str(type(y.grad_fn)) or any("DenseFn" in str(type(f[0])) for f in y.grad_fn.next_functions)
    w, b = (v.value for v in layer.trainable_variables)
    second = []
    for out in (y, torch.relu(x @ w + b)):
        (g,) = torch.autograd.grad((out ** 3).sum(), x, create_graph=True)
        second.append(torch.autograd.grad((g ** 2).sum(), w)[0])
    assert torch.allclose(second[0], second[1], rtol=1e-4, atol=1e-5 * second[1].abs().max().item())
    bad = x.detach().clone()
    bad[0, 0] = float("nan")
    assert layer(bad)[0].isnan().all() and not layer(bad)[1:].isnan().any()


@pytest.mark.parametrize("policy", ["float32", "mixed_bfloat16"])
def test_exported_and_traced_layers_take_any_batch(policy, tmp_path):
    import keras_b200 as keras

    keras.config.set_dtype_policy(policy)
    try:
        i = keras.Input((48,))
        layer = keras.layers.Dense(256, activation="relu")
        model = keras.Model(i, keras.layers.Dense(64)(layer(i)))
    finally:
        keras.config.set_dtype_policy("float32")
    tol = 1e-5 if policy == "float32" else 2e-2  # fp32 sums of 256; two roundings to bf16 a layer
    x = torch.randn(300, 48, device="cuda")
    want = model(x).detach()
    model.export(str(tmp_path / "m"), format="torch_export", verbose=False)
    program = torch.export.load(str(tmp_path / "m" / "serve.pt2")).module()
    with torch.no_grad():
        for v in layer.trainable_variables:  # a trace holds weights as constants
            v._value.requires_grad_(False)
        traced = torch.jit.trace(layer.call, x[:2], check_trace=False)
        for n in (2, 3, 300):
            assert _rel(program(x[:n]).float(), want[:n].double()) < tol, n
            assert _rel(traced(x[:n]).float(), layer.call(x[:n]).double()) < tol, n


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_autocast_reaches_layers_of_any_batch(dtype):
    """The products of a float32 layer are the library's, in the type that the caller asked for, on both sides of the rules for kernels."""
    import keras_b200 as keras

    dense, lstm = keras.layers.Dense(64, activation="relu"), keras.layers.LSTM(16)
    x = torch.randn(300, 12, 48, device="cuda")
    want = dense(x[:, 0]), lstm(x)
    with torch.autocast("cuda", dtype=dtype):
        for n in (8, 300):
            for layer, inputs, ref in ((dense, x[:n, 0], want[0]), (lstm, x[:n], want[1])):
                # one product in 16 bits a step, twelve steps that forget
                assert 1e-5 < _rel(layer(inputs).float(), ref[:n].detach().double()) < 2.0 ** -6


def test_models_in_16_bits_under_autocast_repeat_themselves():
    import keras_b200 as keras

    keras.config.set_dtype_policy("mixed_bfloat16")
    try:
        i = keras.Input((64,))
        model = keras.Model(i, keras.layers.Dense(64)(keras.layers.Dense(64, activation="gelu")(i)))
    finally:
        keras.config.set_dtype_policy("float32")
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.float16):
        x = torch.randn(9, 64, device="cuda")
        first, second = model(x), model(x)
    assert first.dtype == second.dtype and torch.equal(first, second)


# ------------------------------------------------------------------------------------------------ a recorded step that reads a rounded batch
@pytest.mark.parametrize("reader", [None, "dense", "float32", "mixed_float16", "mixed_bfloat16"])
def test_recorded_step_copies_what_it_reads(reader):
    """New batches reach a step whose input only convolutions read in bf16, and one whose input something else reads too.  Each batch has offsets of its
    own, so that a branch that kept the recorded one would take its steps in other directions."""
    import keras_b200 as keras

    def run(graph):
        L = keras.layers
        keras.utils.set_random_seed(6)
        keras.config.set_dtype_policy("mixed_bfloat16")

        def branch(i, dtype=None):
            return L.GlobalAveragePooling2D()(L.ReLU()(L.BatchNormalization(dtype=dtype)(L.Conv2D(32, 1, use_bias=False, dtype=dtype)(i))))

        try:
            i = keras.Input((12, 12, 16))
            parts = [branch(i)]
            if reader:
                parts.append(L.GlobalAveragePooling2D()(i) if reader == "dense" else branch(i, reader))
            model = keras.Model(i, L.Dense(4)(L.Concatenate()(parts) if reader else parts[0]))
        finally:
            keras.config.set_dtype_policy("float32")
        model.compile(keras.optimizers.SGD(0.05), keras.losses.SparseCategoricalCrossentropy(from_logits=True), jit_compile="auto" if graph else False)
        before = [v.value.detach().clone() for v in model.trainable_variables]
        for k in range(9):
            g = torch.Generator(device="cuda").manual_seed(k)
            y = torch.randint(0, 4, (64,), generator=g, device="cuda")
            x = torch.randn(64, 12, 12, 16, generator=g, device="cuda") + 2 * torch.randn(4, 16, generator=g, device="cuda")[y][:, None, None]
            model.train_on_batch(x, y)
        return model, [v.value.detach() - b for v, b in zip(model.trainable_variables, before)]

    (model, recorded), (_, eager) = run(True), run(False)
    step = model._graphed_step
    assert step is not None and step.replays >= 4, getattr(step, "disabled", None)
    assert step.rounded_only == ({0} if reader in (None, "mixed_bfloat16") else set())
    # the distance that each weight went: gradients in bf16, a hundredth apart in two runs
    for a, b in zip(recorded, eager):
        assert _rel(a, b.double()) < 0.1, [_rel(p, q.double()) for p, q in zip(recorded, eager)]


# ------------------------------------------------------------------------------------------------ few classes, running means, BatchNorm sums
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,V,ld", [(1, 2, 2), (128, 10, 10), (777, 37, 40), (513, 21, 24), (65, 63, 63), (33, 8, 8)])
@pytest.mark.parametrize("spread", [True, False])
def test_cross_entropy_of_few_classes(rows, V, ld, dtype, spread):
    from keras_b200.kernels import ops as kops

    g = torch.Generator(device="cuda").manual_seed(rows)
    buf = (torch.randn(rows, ld, generator=g, device="cuda") * 4).to(dtype)
    logits = buf[:, :V].requires_grad_(True)
    if V > 9:
        with torch.no_grad():
            logits[0, 1], logits[0, 2] = float("-inf"), torch.finfo(dtype).min
    labels = torch.randint(3 if V > 9 else 0, V, (rows,), generator=g, device="cuda")
    ref_in = logits.detach().double().requires_grad_(True)
    loss, ref = kops.FusedSoftmaxXent.apply(logits, labels), torch.nn.functional.cross_entropy(ref_in, labels, reduction="none")
    up = torch.rand((), device="cuda").expand(rows) if spread else torch.rand(rows, device="cuda")
    a, = torch.autograd.grad(loss, logits, up)
    b, = torch.autograd.grad(ref, ref_in, up.double())
    # fp32 sums of at most 63 exponentials in full accuracy on the exact inputs; the gradient is rounded once to its type
    assert torch.allclose(loss.double(), ref, atol=2e-6, rtol=5e-7)
    # a probability is exp(v - lse), whose argument of up to 32 is rounded at 2^-20; next to the label it is one less
    assert torch.allclose(a.double(), b, atol=2.0 ** -20, rtol=2.0 ** -19 if dtype == torch.float32 else 2.0 ** -8)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("V", [2, 10, 63])
@pytest.mark.parametrize("bad", [-1, -101, 1 << 40, None])
def test_a_label_that_is_no_class_is_refused(V, dtype, bad):
    """NaN in its row and an error at the next look; -100 is ignored, as by the library."""
    from keras_b200.kernels import ops as kops

    logits = torch.randn(5, V, device="cuda").to(dtype).requires_grad_(True)
    labels = torch.tensor([0, -100, V if bad is None else bad, V - 1, 1], device="cuda")
    loss = kops.FusedSoftmaxXent.apply(logits, labels)
    (grad,) = torch.autograd.grad(loss, logits, torch.ones(5, device="cuda"))
    assert loss.isnan().tolist() == [False, False, True, False, False] and grad[2].isnan().all() and not grad[[0, 1, 3, 4]].isnan().any()
    assert loss[1] == 0 and not grad[1].any()
    with pytest.raises(ValueError, match="label outside"):
        kops.check_labels()
    kops.check_labels()
    kops.FusedSoftmaxXent.apply(logits, labels.clamp(0, V - 1))
    torch.cuda.synchronize()
    kops.check_labels()


@pytest.mark.parametrize("recorded", [True, False])
def test_training_on_a_label_that_is_no_class_raises(recorded):
    import keras_b200 as keras

    model = keras.Sequential([keras.Input((8,)), keras.layers.Dense(5)])
    model.compile("sgd", keras.losses.SparseCategoricalCrossentropy(from_logits=True), jit_compile="auto" if recorded else False)
    x, y = torch.randn(16, 8, device="cuda"), torch.arange(16, device="cuda") % 5
    for _ in range(6):
        model.train_on_batch(x, y)
    assert not recorded or model._graphed_step.replays
    with pytest.raises(ValueError, match="label outside"):
        model.train_on_batch(x, y + 1)
    with pytest.raises(ValueError, match="label outside"):
        model.test_on_batch(x, y + 1)
    with pytest.raises(ValueError, match="label outside"):
        model.fit(x, y + 1, batch_size=16, epochs=1, verbose=0)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("V,ld", [(2, 2), (10, 10), (37, 40), (63, 63), (64, 64), (300, 304), (2049, 2056)])
@pytest.mark.parametrize("layout", ["rows", "columns", "expected"])
def test_cross_entropy_second_derivatives(V, ld, dtype, layout):
    """Rows with a pitch, rows that have to be copied, and a gradient that was made ahead."""
    import contextlib

    from keras_b200.kernels import ops as kops

    g = torch.Generator(device="cuda").manual_seed(V)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(dtype)  # noqa: E731
    logits = (rnd(V, 6).t() if layout == "columns" else rnd(6, ld)[:, :V]).requires_grad_(True)
    labels = torch.randint(0, V, (6,), generator=g, device="cuda")
    up = torch.rand(6, generator=g, device="cuda").requires_grad_(True)
    with kops.gradient_follows() if layout == "expected" else contextlib.nullcontext():
        kops.expect_upstream(lambda n: 1.0 / n)
        loss = kops.FusedSoftmaxXent.apply(logits, labels)
    exact = [t.detach().double().requires_grad_(True) for t in (logits, up)]
    want = torch.nn.functional.cross_entropy(exact[0], labels, reduction="none")
    probe = rnd(6, V)
    both = []
    for value, z, u in ((loss, logits, up), (want, *exact)):
        (first,) = torch.autograd.grad((value * u).sum(), z, create_graph=True)
        both.append((first, *torch.autograd.grad((first * probe.to(first.dtype)).sum(), (z, u))))
    # three chains of fp32 operations, rounded to the type of the logits where they leave for them and back
    for a, b in zip(*both):
        assert _rel(a.detach(), b.detach()) < (1e-5 if dtype == torch.float32 else 2.0 ** -6)


@pytest.mark.parametrize("V", [2, 37, 63])
def test_cross_entropy_of_few_classes_in_the_type_of_its_logits(V):
    """The op's values have it, rounded once; a loss object's are float32 whatever it is given, and a subclass is given float32."""
    import keras_b200 as keras

    class Own(keras.losses.SparseCategoricalCrossentropy):
        def call(self, y_true, y_pred):
            seen.append(y_pred.dtype)
            return super().call(y_true, y_pred)

    seen = []
    logits, labels = torch.randn(65, V, device="cuda").bfloat16(), torch.randint(0, V, (65,), device="cuda")
    want = torch.nn.functional.cross_entropy(logits.double(), labels, reduction="none")
    for fn in (keras.ops.sparse_categorical_crossentropy, keras.losses.sparse_categorical_crossentropy):
        values = fn(labels, logits, from_logits=True)
        assert values.dtype == torch.bfloat16 and torch.allclose(values.double(), want, rtol=2.0 ** -8, atol=1e-6)
        assert fn(labels, logits.float(), from_logits=True).dtype == torch.float32
    for kind in (keras.losses.SparseCategoricalCrossentropy, Own):
        loss = kind(from_logits=True, reduction=None)(labels, logits)
        assert loss.dtype == torch.float32 and torch.allclose(loss.double(), want, rtol=5e-7, atol=2e-6)
    assert seen == [torch.float32]


def test_running_means_round_as_their_operations():
    import keras_b200 as keras

    mean = keras.metrics.Mean()
    total, count = torch.zeros((), device="cuda"), torch.zeros((), device="cuda")
    assert float(mean.result()) == 0.0
    for k, w in enumerate((3, 64, 0.1, 7)):
        value = torch.randn((), device="cuda", generator=torch.Generator(device="cuda").manual_seed(k))
        mean.update_state(value, sample_weight=w)
        total, count = total + value * w, count + w
        assert torch.equal(mean.result(), total / count) and mean.result().device.type == "cuda"
    mean.reset_state()
    assert float(mean.total.value) == float(mean.count.value) == float(mean.result()) == 0.0
    mean.update_state(torch.tensor([1.0, 3.0], device="cuda"))
    assert float(mean.result()) == 2.0
    mean.reset_state()
    mean.update_state(torch.tensor(float("nan"), device="cuda"), sample_weight=2)
    assert torch.isnan(mean.result())


def test_a_running_mean_of_given_numbers_has_gradients():
    import keras_b200 as keras

    mean = keras.metrics.Mean()
    total, count = (torch.tensor(v, device="cuda", requires_grad=True) for v in (3.0, 2.0))
    grads = torch.autograd.grad(mean.stateless_result([total, count]), (total, count))
    assert [float(g) for g in grads] == [0.5, -0.75]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", [(2, 3, 3, 8), (4, 9, 9, 96), (24, 18, 18, 384), (32, 32, 32, 256)])
@pytest.mark.parametrize("residual", [False, True])
def test_batch_norm_backward_twice_and_into_the_arena(shape, dtype, residual):
    """The sums that the forward pass clears serve one backward pass; another one, and gradients of their own, have theirs."""
    from keras_b200.kernels import ops as kops
    from keras_b200.kernels import shadow

    g = torch.Generator(device="cuda").manual_seed(1)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    C = shape[-1]
    x, r = rnd(*shape).to(dtype).requires_grad_(True), (rnd(*shape).to(dtype).requires_grad_(True) if residual else None)
    gamma, beta = (1 + 0.1 * rnd(C)).requires_grad_(True), rnd(C).requires_grad_(True)
    up = rnd(*shape).to(dtype)

    def forward():
        return kops.FusedBatchNormAct.apply(x, gamma, beta, r, torch.zeros(C, device="cuda"), torch.ones(C, device="cuda"), 0.9, 1e-3, True)

    inputs = [t for t in (x, gamma, beta, r) if t is not None]
    y = forward()
    own = [torch.autograd.grad(y, inputs, up, retain_graph=True) for _ in range(2)]  # of one forward pass: another's mean may turn a rectifier over
    gamma.grad, beta.grad = torch.full((C,), 2.0, device="cuda"), torch.full((C,), -1.0, device="cuda")
    rest = [t for t in (x, r) if t is not None]
    with shadow.arena_backward():
        arena = [torch.autograd.grad(y, rest, up, retain_graph=k == 0) for k in range(2)]
    tol = 2e-5 if dtype == torch.float32 else 2.0 ** -7  # sums of up to 32768 products in fp32, added in any order; one rounding of dx
    for k in range(2):
        for a, b in zip([own[k][0]] + list(own[k][3:]), own[0][:1] + own[0][3:]):
            assert _rel(a, b.double()) < tol
        assert _rel(own[k][1], own[0][1].double()) < 1e-5 and _rel(own[k][2], own[0][2].double()) < 1e-5
        for a, b in zip(arena[k], own[0][:1] + own[0][3:]):
            assert _rel(a, b.double()) < tol
    assert _rel(gamma.grad - 2.0, 2 * own[0][1].double()) < 1e-4 and _rel(beta.grad + 1.0, 2 * own[0][2].double()) < 1e-4
    ex = [t.detach().double().requires_grad_(True) for t in inputs]
    flat = ex[0].reshape(-1, C)
    z = torch.nn.functional.batch_norm(flat, None, None, ex[1], ex[2], True, 0.0, 1e-3).reshape(shape) + (ex[3] if residual else 0)
    for a, b in zip(own[0], torch.autograd.grad(z * (y.detach() > 0), ex, up.double())):
        assert _rel(a, b) < (1e-4 if dtype == torch.float32 else 2.0 ** -6)


# ------------------------------------------------------------------------------------------------ slices of K, gradients in place
@pytest.mark.parametrize("M,K,N", [(128, 64, 4096), (130, 256, 8009), (2664, 512, 8009), (4096, 512, 8009), (300, 768, 12000), (2664, 512, 512), (512, 384, 384)])
def test_dense_gradients_in_slices(M, K, N):
    from keras_b200.kernels import gemm

    g = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16().requires_grad_(True)
    w = (torch.randn(K, N, generator=g, device="cuda") * K ** -0.5).bfloat16().requires_grad_(True)
    up = torch.randn(M, N, generator=g, device="cuda").bfloat16()
    dx, dw = torch.autograd.grad(gemm.GemmFn.apply(x, w, None, None, None), (x, w), up)
    # exact products of bf16, fp32 sums in any order, one rounding to bf16
    assert _rel(dx, up.double() @ w.detach().double().t()) < 2.0 ** -8
    assert _rel(dw, x.detach().double().t() @ up.double()) < 2.0 ** -8
    gemm.check_errors()


@pytest.mark.parametrize("M,K,N", [(128, 64, 4096), (130, 256, 8009), (2664, 512, 8009), (300, 768, 12000), (31, 72, 5000), (1900, 512, 512), (1024, 1024, 3072),
                                   (2047, 768, 2304), (5000, 2048, 2560)])
def test_dense_gradients_repeat_bit_for_bit(M, K, N):
    """Slices of a vocabulary are added in order; weight gradients over fewer than 2048 rows, or whose tiles fill half of the chip, are one slice."""
    from keras_b200.kernels import gemm

    g = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16().requires_grad_(True)
    w = (torch.randn(K, N, generator=g, device="cuda") * K ** -0.5).bfloat16().requires_grad_(True)
    up = torch.randn(M, N, generator=g, device="cuda").bfloat16()
    y = gemm.GemmFn.apply(x, w, None, None, None)
    first = torch.autograd.grad(y, (x, w), up, retain_graph=True)
    assert _rel(first[0], up.double() @ w.detach().double().t()) < 2.0 ** -8  # exact products, fp32 sums, one rounding
    for _ in range(5):
        again = torch.autograd.grad(y, (x, w), up, retain_graph=True)
        assert torch.equal(first[0], again[0])
        assert M >= 2048 and K * N < 1 << 21 or torch.equal(first[1], again[1])
    gemm.check_errors()


def test_embedding_gradient_goes_into_the_arena():
    import keras_b200 as keras
    from keras_b200.kernels import shadow

    keras.config.set_dtype_policy("mixed_bfloat16")
    try:
        layer = keras.layers.Embedding(50, 64)
        layer.build((None, 7))
    finally:
        keras.config.set_dtype_policy("float32")
    ids = torch.randint(-3, 50, (9, 7), device="cuda", dtype=torch.int32)
    table = layer._embeddings._value
    up = torch.randn(9, 7, 64, device="cuda").bfloat16()
    want = torch.zeros(50, 64, device="cuda").index_add_(0, ids.long().reshape(-1) % 50, up.float().reshape(-1, 64))
    (own,) = torch.autograd.grad(layer(ids), table, up)
    table.grad = torch.full_like(table, 2.0)
    y = layer(ids)
    with shadow.arena_backward():
        y.backward(up)
    assert _rel(own, want.double()) < 1e-6 and _rel(table.grad - 2.0, want.double()) < 1e-5


@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 1024), (1000, 264), (2664, 2048)])
def test_gelu_of_a_matrix(rows, cols):
    from keras_b200.kernels import ops as kops

    z = (torch.randn(rows, cols, device="cuda") * 4).bfloat16()
    z[0, :4] = torch.tensor([float("inf"), float("-inf"), float("nan"), 0.0])
    y, want = kops.gelu(z), z.double() * torch.special.erfc(z.double() * -(0.5 ** 0.5)) / 2  # without the cancellation of 1 + erf
    assert torch.equal(y[0, :4].isnan(), want[0, :4].isnan()) and y[0, 0] == float("inf") and y[0, 3] == 0
    assert torch.allclose(y.double(), want, rtol=2.0 ** -8, atol=1e-36, equal_nan=True)  # one rounding; the distribution function within 2.5e-6


@pytest.mark.parametrize("policy", ["float32", "mixed_bfloat16"])
def test_gradient_hooks_see_the_gradients_of_a_training_step(policy):
    import keras_b200 as keras

    def steps(hooked):
        L = keras.layers
        keras.utils.set_random_seed(8)
        keras.config.set_dtype_policy(policy)
        try:
            i = keras.Input((40,), dtype="int32")
            h = L.Embedding(30, 32)(i)
            h = L.LSTM(16)(h) if policy == "float32" else L.GlobalAveragePooling1D()(L.LayerNormalization()(h))
            model = keras.Model(i, L.Dense(64)(L.Dense(64, activation="relu")(h)))
        finally:
            keras.config.set_dtype_policy("float32")
        model.compile(keras.optimizers.SGD(0.1), keras.losses.SparseCategoricalCrossentropy(from_logits=True), run_eagerly=True)
        seen = {}
        if hooked:
            for v in model.trainable_variables:
                v._value.register_hook(lambda g, _p=v.path: seen.setdefault(_p, []).append(None if g is None else g.detach().clone()))
        g = torch.Generator(device="cuda").manual_seed(1)
        for _ in range(4):
            model.train_on_batch(torch.randint(0, 30, (64, 40), generator=g, device="cuda", dtype=torch.int32), torch.randint(0, 64, (64,), generator=g, device="cuda"))
        return model, seen

    model, seen = steps(True)
    assert set(seen) == {v.path for v in model.trainable_variables}
    assert all(len(gs) == 4 and all(g is not None and g.any() for g in gs) for gs in seen.values()), {p: [g is not None for g in gs] for p, gs in seen.items()}
    for a, b in zip(model.trainable_variables, steps(False)[0].trainable_variables):
        assert _rel(a.value, b.value.detach().double()) < (1e-5 if policy == "float32" else 1e-2)  # gradients in fp32 either way; rounded to bf16 on their way to a hook
