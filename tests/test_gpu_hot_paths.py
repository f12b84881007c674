"""The variants a dispatch rule chooses between, each at the sizes where it can go wrong (needs a B200)."""

import gc

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,V,ld", [(1, 64, 64), (77, 64, 64), (513, 65, 72), (100, 100, 100), (33, 129, 136), (7, 1000, 1000), (19, 2047, 2047),
                                       (9, 2048, 2048), (5, 2049, 2056), (5, 5001, 5001)])
def test_cross_entropy_of_narrow_and_wide_rows(rows, V, ld, dtype):
    from keras_b200.kernels import ops as kops

    torch.manual_seed(V)
    buf = (torch.randn(rows, ld, device="cuda") * 3).to(dtype)
    if V > 70:
        buf[:, 3:17] = float("-inf")  # masked classes
        buf[0, 17:20] = torch.finfo(dtype).min  # masks of the lowest value
    logits = buf[:, :V].detach().requires_grad_(True)
    labels = torch.randint(20, V, (rows,), device="cuda")
    if rows > 2:
        labels[1] = -1  # not a class: no loss, no gradient
    loss = kops.FusedSoftmaxXent.apply(logits, labels)
    g = torch.rand(rows, device="cuda")
    loss.backward(g)
    ref_in = logits.detach().double().requires_grad_(True)
    valid = labels >= 0
    ref = torch.nn.functional.cross_entropy(ref_in, labels, reduction="none", ignore_index=-1)
    ref.backward(g.double())
    assert torch.equal(loss == 0, ~valid)
    # fp32 sums of at most 2049 exponentials on the exact inputs; the gradient is rounded once to its type
    assert torch.allclose(loss.double(), ref, atol=1e-5, rtol=1e-5)
    assert torch.allclose(logits.grad.double(), ref_in.grad, atol=1e-6, rtol=1e-5 if dtype == torch.float32 else 2.0 ** -8)


GEMM_VARIANTS = {1: "one tile a CTA", 2: "persistent", 3: "CTA pairs"}


@pytest.mark.parametrize("variant", sorted(GEMM_VARIANTS))
@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (264, 520, 384), (264, 520, 392), (16392, 264, 200), (264, 520, 1000), (136, 1000, 72), (2664, 512, 520), (2049 * 8, 264, 136)])
def test_gemm_variants_agree_with_the_product_in_64_bits(M, N, K, variant):
    from keras_b200.kernels import ops as K_

    lib = K_._lib()
    torch.manual_seed(M + N)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for a_mn, b_mn in [(0, 1), (0, 0), (1, 1), (1, 0)]:
        a = torch.randn((K, M) if a_mn else (M, K), device="cuda").bfloat16()
        b = torch.randn((K, N) if b_mn else (N, K), device="cuda").bfloat16()
        bias = torch.randn(N, device="cuda")
        ref = (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double()
        for split, fp32, add in [(1, 0, False), (1, 1, False), (3, 1, False), (-2, 1, True)]:
            if variant == 1 and split not in (1, -1):
                continue
            c = torch.full((M, N), 2.0, device="cuda") if add else torch.zeros((M, N), device="cuda", dtype=torch.float32 if fp32 else torch.bfloat16)
            with_bias = split == 1
            code = lib.kb200_gemm_bf16_run(K_._p(a), K_._p(b), K_._p(c), K_._p(bias if with_bias else None), K_._i(M), K_._i(N), K_._i(K),
                                           K_._ll(a.stride(0)), K_._ll(b.stride(0)), K_._ll(N), K_._i(a_mn), K_._i(b_mn), K_._i(1 if with_bias else 0),
                                           K_._i(fp32), K_._i(0), K_._i(split), K_._i(variant), K_._p(err), K_._stream())
            K_._check(code, "gemm_bf16")
            want = torch.relu(ref + bias) if with_bias else ref + 2.0 if add else ref
            rel = ((c.double() - want).norm() / want.norm()).item()
            # fp32 sums of K exact products (2^-24 each), one rounding to bf16 (2^-9)
            assert rel < (2.0 ** -17 if fp32 else 2.0 ** -8), (a_mn, b_mn, split, fp32, rel)
            assert int(err.item()) == 0


@pytest.mark.parametrize("B,T,U,F", [(1, 1, 4, 3), (3, 7, 20, 5), (64, 5, 256, 16), (37, 9, 72, 8), (200, 3, 512, 8), (300, 2, 640, 4)])
@pytest.mark.parametrize("reverse,sequence", [(False, True), (True, True), (False, False)])
def test_lstm_sequence_against_the_steps_in_64_bits(B, T, U, F, reverse, sequence):
    from keras_b200.kernels import gemm, lstm

    g = torch.Generator(device="cuda").manual_seed(B + U)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    args = [rnd(B, T, 4 * U), rnd(4 * U), 0.5 * rnd(B, U), rnd(B, U), rnd(U, 4 * U) * U ** -0.5]
    mine = [a.clone().requires_grad_(True) for a in args]
    exact = [a.double().requires_grad_(True) for a in args]
    out, h, c = lstm.run(*mine, reverse, sequence)
    want, hw, cw = lstm._composed(*exact, reverse)
    up = [rnd(B, T, U), rnd(B, U), rnd(B, U)]
    loss = (h * up[1]).sum() + (c * up[2]).sum() + ((out * up[0]).sum() if sequence else 0)
    ref = (hw * up[1]).sum() + (cw * up[2]).sum() + ((want * up[0]).sum() if sequence else 0)
    loss.backward()
    ref.backward()
    gemm.check_errors()
    # fp32 sums over U terms a step and up to B * T in the weight gradient, a few steps deep
    rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()  # noqa: E731
    assert rel(h, hw) < 3e-6 and rel(c, cw) < 3e-6 and (not sequence or rel(out, want) < 3e-6)
    for a, b in zip(mine, exact):
        assert rel(a.grad, b.grad) < 1e-5
    with torch.no_grad():
        out2, h2, c2 = lstm.run(*mine, reverse, sequence)
    assert torch.equal(h2, h) and torch.equal(c2, c)


@pytest.mark.parametrize("B,T,U", [(3, 1, 20), (64, 6, 256), (300, 4, 640)])
@pytest.mark.parametrize("reverse", [False, True])
def test_lstm_keeps_gates_only_for_a_backward_pass(B, T, U, reverse, monkeypatch):
    """Trainable weights without gradients: no gates, no cell states, the same result bit for bit (several row tiles a group at B = 300)."""
    from keras_b200.kernels import lstm

    g = torch.Generator(device="cuda").manual_seed(U)
    args = [torch.randn(s, generator=g, device="cuda") for s in ((B, T, 4 * U), (4 * U,), (B, U), (B, U))]
    args.append((torch.randn((U, 4 * U), generator=g, device="cuda") * U ** -0.5).requires_grad_(True))
    launched, plain = [], lstm._launch
    monkeypatch.setattr(lstm, "_launch", lambda *a: launched.append(a) or plain(*a))
    recorded = lstm.run(*args, reverse, True)
    with torch.no_grad():
        bare = lstm.run(*args, reverse, True)
    assert [a[10] is None and a[11] is None for a in launched] == [False, True]
    assert all(torch.equal(a, b) for a, b in zip(recorded, bare))


def test_lstm_layer_routes_and_second_derivatives():
    import keras_b200 as keras
    from keras_b200.kernels import lstm

    keras.utils.set_random_seed(0)
    layer = keras.layers.LSTM(24, return_sequences=True)
    x = torch.randn(5, 6, 8, device="cuda", requires_grad=True)
    y = layer(x)
    assert "LstmSequence" in str(type(y.grad_fn)) or any("LstmSequence" in str(type(f[0])) for f in y.grad_fn.next_functions)
    weights = [v.value for v in layer.trainable_variables]
    z = torch.matmul(x, weights[0])
    zero = torch.zeros(5, 24, device="cuda")
    want = lstm._composed(z, weights[2], zero, zero, weights[1], False)[0]
    assert torch.allclose(y, want, atol=2e-6)
    second = []
    for out in (y, want):
        (g,) = torch.autograd.grad((out ** 2).sum(), x, create_graph=True)
        second.append(torch.autograd.grad((g ** 2).sum(), weights[1])[0])
    assert torch.allclose(second[0], second[1], rtol=1e-4, atol=1e-5 * second[1].abs().max().item())
    # function transforms keep to the composed operations
    frozen = x.detach()
    batched = torch.func.vmap(lambda s: layer(s.unsqueeze(0)).squeeze(0))(frozen)
    assert torch.allclose(batched, want, atol=2e-6)


def _attention_in_64_bits(q, k, v, scale, causal, mask):
    """[B, T, heads, head size]; masked scores are a finite negative, as the layers define them."""
    q, k, v = (t.double().transpose(1, 2) for t in (q, k, v))
    k, v = (t.repeat_interleave(q.shape[1] // t.shape[1], dim=1) for t in (k, v))
    s = torch.matmul(q, k.transpose(-1, -2)) * scale
    if causal:
        s = s.masked_fill(torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    if mask is not None:
        s = s.masked_fill(~mask, -1e30)
    return torch.matmul(torch.softmax(s, dim=-1), v).transpose(1, 2)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Tq,Tk,H,Hkv", [(2, 1, 1, 2, 2), (3, 77, 77, 4, 2), (1, 128, 129, 2, 1), (2, 129, 300, 2, 2), (1, 256, 256, 6, 2), (2, 333, 333, 3, 3),
                                           (1, 700, 65, 2, 2), (1, 1024, 1024, 2, 1)])
@pytest.mark.parametrize("kind", ["none", "causal", "rows", "keys", "causal+keys"])
def test_attention_against_64_bits(B, Tq, Tk, H, Hkv, D, kind):
    from keras_b200.kernels import attention

    g = torch.Generator(device="cuda").manual_seed(Tq + Tk)
    q, k, v = (torch.randn(s, generator=g, device="cuda").bfloat16() for s in ((B, Tq, H, D), (B, Tk, Hkv, D), (B, Tk, Hkv, D)))
    q = q * 4  # peaked rows: the maximum moves from block to block
    mask = None
    if kind == "rows":
        mask = torch.rand((B, 1, Tq, Tk), generator=g, device="cuda") < 0.7
        mask[:, :, Tq // 2:Tq // 2 + 3] = False  # rows without any key attend uniformly
        mask[:, :, :, : min(130, Tk // 2)] &= torch.rand((B, 1, Tq, 1), generator=g, device="cuda") < 0.5  # whole blocks without a key
    elif "keys" in kind:
        mask = (torch.arange(Tk, device="cuda") < torch.randint(1, Tk + 1, (B, 1), generator=g, device="cuda"))[:, None, None, :]
    causal = "causal" in kind
    out = attention.flash_attention(q, k, v, mask, D ** -0.5, causal)
    assert out is not None
    attention.check_errors()
    if causal and mask is not None:
        mask, causal = mask & torch.ones((Tq, Tk), dtype=torch.bool, device="cuda").tril(), False
    want = _attention_in_64_bits(q, k, v, D ** -0.5, causal, mask)
    # probabilities and result are rounded to bf16 once each (2^-9), the sums are fp32
    rel = ((out.double() - want).norm() / want.norm()).item()
    assert rel < 2.0 ** -8, rel
    assert (out.double() - want).abs().max().item() < 0.03 * v.abs().max().item()


@pytest.mark.parametrize("D,T", [(64, 77), (128, 300), (64, 512)])
def test_attention_with_masked_rows_and_keys(D, T):
    from keras_b200.kernels import attention

    g = torch.Generator(device="cuda").manual_seed(T)
    q, k, v = (torch.randn((3, T, 4, D), generator=g, device="cuda").bfloat16() for _ in range(3))
    lengths = torch.tensor([[T], [1], [T // 2]], device="cuda")
    real = torch.arange(T, device="cuda") < lengths
    out = attention.forward(q, k, v, D ** -0.5, False, real[:, None, None, :].expand(3, 4, T, T), real)[0]
    attention.check_errors()
    want = _attention_in_64_bits(q, k, v, D ** -0.5, False, real[:, None, :, None] & real[:, None, None, :])
    assert ((out.double() - want).norm() / want.norm()).item() < 2.0 ** -8


@pytest.mark.parametrize("masks", ["both", "query+key", "three", "query only", "of integers"])
def test_attention_layer_with_padding(masks):
    """Rows and keys that are padding: the layer against itself with their product as an explicit mask."""
    import keras_b200 as keras
    from keras_b200.kernels import attention

    T, S = 77, 77 if masks == "both" else 130
    layer = keras.layers.MultiHeadAttention(4, 64, dtype="bfloat16")
    g = torch.Generator(device="cuda").manual_seed(5)
    q = torch.randn((3, T, 256), generator=g, device="cuda").bfloat16()
    v = q if masks == "both" else torch.randn((3, S, 256), generator=g, device="cuda").bfloat16()
    rows = torch.arange(T, device="cuda") < torch.tensor([[T], [1], [T // 2]], device="cuda")
    keys = rows if masks == "both" else torch.arange(S, device="cuda") < torch.tensor([[S], [70], [3]], device="cuda")
    other = torch.rand((3, S), generator=g, device="cuda") < 0.8
    given, seen = {"both": ({"value_mask": keys}, keys), "query+key": ({"key_mask": keys}, keys), "of integers": ({"value_mask": keys.to(torch.int32)}, keys),
                   "three": ({"value_mask": keys, "key_mask": other}, keys & other), "query only": ({}, torch.ones_like(keys))}[masks]
    with torch.no_grad():
        want = layer(q, v, attention_mask=rows[:, :, None] & seen[:, None, :])
        calls, plain = [], attention.forward
        attention.forward = lambda *a, **k: calls.append(a) or plain(*a, **k)
        try:
            got = layer(q, v, query_mask=rows, **given)
        finally:
            attention.forward = plain
        attention.check_errors()
        assert torch.equal(got, want) and len(calls) == 1
        assert (calls[0][-1] is rows) == (masks in ("both", "query+key", "three"))
    # training keeps the product, for the library
    out = layer(q.clone().requires_grad_(True), v, query_mask=rows, **given)
    assert ((out.double() - want.double()).norm() / want.double().norm()).item() < 2.0 ** -6


def _uniform_rows(keras, dtype, causal, biased, device):
    g = torch.Generator(device=device).manual_seed(9)
    q, k, v, dy = (torch.randn((2, 40, 4, 64), generator=g, device=device).to(dtype) for _ in range(4))
    mask = torch.rand((2, 1, 40, 40), generator=g, device=device) < 0.5
    mask[..., 0] = True
    mask[:, :, 3] = mask[1, :, 20:25] = False
    bias = torch.randn((4, 40, 40), generator=g, device=device).to(dtype) if biased else None
    args = [t.requires_grad_(True) for t in (q, k, v)]
    out = keras.ops.dot_product_attention(*args, bias=bias, mask=mask, is_causal=causal)
    grads = torch.autograd.grad(out, args, dy)
    with torch.no_grad():
        inferred = keras.ops.dot_product_attention(q, k, v, bias=bias, mask=mask, is_causal=causal)
    seen = mask & torch.ones((40, 40), dtype=torch.bool, device=device).tril() if causal else mask
    empty = ~seen.any(-1, keepdim=True)
    exact = [t.detach().double().requires_grad_(True) for t in args]
    qe, ke, ve = (t.transpose(1, 2) for t in exact)
    s = torch.matmul(qe, ke.transpose(-1, -2)) / 8 + (bias.double() if biased else 0)
    s = s.masked_fill(~seen, -1e30).masked_fill(empty, 0.0)
    want = torch.matmul(torch.softmax(s, -1), ve).transpose(1, 2)
    bound = {torch.bfloat16: 2.0 ** -6, torch.float16: 2.0 ** -9, torch.float32: 1e-5}[dtype]  # a few roundings of scores and probabilities
    for a, e in zip([out, inferred, *grads], [want, want, *torch.autograd.grad(want, exact, dy.double())]):
        assert ((a.double() - e).norm() / e.norm()).item() < bound
    rows = empty.squeeze(-1).expand(2, 4, 40).transpose(1, 2)
    assert torch.allclose(out[rows].float(), v.float().mean(1, keepdim=True).expand(v.shape)[rows], atol=0.02)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("causal,biased", [(False, False), (True, False), (False, True)])
def test_attention_of_rows_without_a_key_is_uniform_in_training_too(dtype, causal, biased):
    import keras_b200 as keras

    _uniform_rows(keras, dtype, causal, biased, "cuda")


def _broadcast_masks(keras, dtype, device, T, S, H, D):
    """Masks and biases of one column, one row or one head, with and without gradients, against 64 bits."""
    g = torch.Generator(device=device).manual_seed(T * S)
    q = torch.randn((3, T, H, D), generator=g, device=device).to(dtype)
    k, v = (torch.randn((3, S, H, D), generator=g, device=device).to(dtype) for _ in range(2))
    for shape in ((3, 1, T, 1), (3, 1, 1, S), (1, 1, T, 1), (T, 1), (1, 1, 1, 1), (3, H, 1, S)):
        for kind in ("mask", "bias"):
            t = torch.randn(shape, generator=g, device=device)
            given = t > -0.5 if kind == "mask" else t.to(dtype)
            s = torch.matmul(q.double().transpose(1, 2), k.double().permute(0, 2, 3, 1)) * D ** -0.5
            if kind == "mask":
                empty = ~given.expand(torch.broadcast_shapes(given.shape, (T, S))).any(-1, keepdim=True)
                s = s.masked_fill(~given, -1e30).masked_fill(empty, 0.0)
            else:
                s = s + given.double()
            want = torch.matmul(torch.softmax(s, -1), v.double().transpose(1, 2)).transpose(1, 2)
            with torch.no_grad():
                outs = [keras.ops.dot_product_attention(q, k, v, **{kind: given})]
            args = [x.clone().requires_grad_(True) for x in (q, k, v)]
            outs.append(keras.ops.dot_product_attention(*args, **{kind: given}))
            outs[-1].backward(torch.ones_like(outs[-1]))
            bound = {torch.bfloat16: 2.0 ** -6, torch.float16: 2.0 ** -9, torch.float32: 1e-5}[dtype]
            for out in outs:
                assert ((out.double() - want).norm() / want.norm()).item() < bound, (shape, kind)
            assert all(a.grad.isfinite().all() for a in args)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("T,S,H,D", [(16, 12, 1, 32), (254, 284, 2, 64), (181, 181, 4, 32), (40, 64, 2, 40)])
def test_attention_under_broadcast_masks_and_biases(dtype, T, S, H, D):
    import keras_b200 as keras

    _broadcast_masks(keras, dtype, "cuda", T, S, H, D)


def test_attention_keeps_a_nan_to_the_rows_that_see_it():
    from keras_b200.kernels import attention

    for bad in (0, 7, 70, 129):  # exponentials on either pipe, both halves of a block, the second block
        q, k, v = (torch.randn((1, 200, 2, 64), device="cuda").bfloat16() for _ in range(3))
        k[0, bad, 0, 3] = float("nan")
        out = attention.forward(q, k, v, 0.125, True)[0]
        assert torch.equal(out.isnan().any(-1)[0, :, 0], torch.arange(200, device="cuda") >= bad) and not out[:, :, 1].isnan().any()


def test_attention_strides_and_refusals():
    from keras_b200.kernels import attention

    g = torch.Generator(device="cuda").manual_seed(3)
    qkv = torch.randn((2, 200, 3, 4, 64), generator=g, device="cuda").bfloat16()
    q, k, v = qkv.unbind(2)  # rows of another pitch
    wide = torch.rand((2, 4, 200, 512), generator=g, device="cuda") < 0.6
    for mask in (wide[..., 7:207], wide[..., ::2][..., :200], wide[:1, :1, :, :1], wide[0, 0, :, 3:203].to(torch.int32)):
        out = attention.flash_attention(q, k, v, mask, 0.125, False)
        want = _attention_in_64_bits(q, k, v, 0.125, False, torch.broadcast_to(mask != 0, (2, 4, 200, 200)))
        assert ((out.double() - want).norm() / want.norm()).item() < 2.0 ** -8
    assert attention.flash_attention(q, k, v, None, -0.125, False) is None  # a negative scale turns the maximum around
    assert attention.flash_attention(q[..., :40], k[..., :40], v[..., :40], None, 0.125, False) is None
    assert attention.flash_attention(q.float(), k.float(), v.float(), None, 0.125, False) is None
    assert attention.flash_attention(q.detach().requires_grad_(True), k, v, wide[..., :200], 0.125, False) is None


def test_attention_leaves_broadcast_operands_to_the_library():
    """Keys and values of fewer batch elements (or heads) than the query's: the kernel would read behind them."""
    import keras_b200 as keras
    from keras_b200.kernels import attention

    g = torch.Generator(device="cuda").manual_seed(11)
    q, k, v = (torch.randn((b, 40, 4, 64), generator=g, device="cuda").bfloat16() for b in (3, 1, 1))
    mask = torch.rand((3, 1, 40, 40), generator=g, device="cuda") < 0.7
    mask[..., 0] = True
    with torch.no_grad():
        for m in (mask, None):
            assert attention.flash_attention(q, k, v, m, 0.125, False) is None
            out = keras.ops.dot_product_attention(q, k, v, mask=m)
            want = _attention_in_64_bits(q, k, v, 0.125, False, m)
            assert ((out.double() - want).norm() / want.norm()).item() < 2.0 ** -7
        three = k.expand(3, 40, 4, 64)
        for keys, values in ((three, v), (k, v.expand(3, 40, 4, 64)), (three, three[:, :, :2]), (three[:, :, :2], three), (three, three[:, :30])):
            assert attention.flash_attention(q, keys, values, mask, 0.125, False) is None
        assert attention.flash_attention(q[:1], three, three, None, 0.125, False) is None
        assert attention.flash_attention(q, three[:, :, :0], three[:, :, :0], None, 0.125, False) is None


def _bf16_model(vocab=300, d=64):
    import keras_b200 as keras

    old = keras.config.dtype_policy()
    keras.config.set_dtype_policy("mixed_bfloat16")
    try:
        x = keras.Input((16, d))
        return keras.Model(x, keras.layers.Dense(vocab)(keras.layers.Dense(d, activation="relu")(x)))
    finally:
        keras.config.set_dtype_policy(old)


def _plain(model, x):
    h = x.bfloat16()
    for i, layer in enumerate(model.layers[1:]):
        h = torch.matmul(h, layer.kernel.value.bfloat16()) + layer.bias.value.bfloat16()
        h = torch.relu(h) if i == 0 else h
    return h


def _agrees(model, x):
    with torch.no_grad():
        return torch.allclose(model(x, training=False).float(), _plain(model, x).float(), atol=0.05, rtol=0.02)


@pytest.mark.parametrize("vocab", [300, 301, 304])
def test_inference_follows_every_change_of_its_weights(vocab):
    """Also those that no version counter shows: writes through ``data``, replays of a recorded update, the fused optimizer."""
    import keras_b200 as keras

    keras.utils.set_random_seed(0)
    model = _bf16_model(vocab)
    x = torch.randn(8, 16, 64, device="cuda")
    first, second = (layer.kernel for layer in model.layers[1:])
    assert all(_agrees(model, x) for _ in range(3))
    first.assign(torch.randn(64, 64, device="cuda") * 0.1)
    assert all(_agrees(model, x) for _ in range(3))
    with torch.no_grad():
        second.value.mul_(2.0)
    assert all(_agrees(model, x) for _ in range(3))
    second.value.data.mul_(-1.5)
    assert all(_agrees(model, x) for _ in range(3))
    model.set_weights([w * 0.5 for w in model.get_weights()])
    assert all(_agrees(model, x) for _ in range(3))
    gc.collect()  # a recorded step of an earlier model, released during a capture, would invalidate it
    update = torch.cuda.CUDAGraph()
    with torch.no_grad(), torch.cuda.graph(update):
        first.value.mul_(-1.25)
    for _ in range(3):
        update.replay()
        assert all(_agrees(model, x) for _ in range(2))
    model.compile(optimizer=keras.optimizers.SGD(0.5, momentum=0.9), loss="mse")
    y = torch.randn(8, 16, vocab, device="cuda")
    for _ in range(6):
        model.train_on_batch(x, y)
        assert all(_agrees(model, x) for _ in range(2))


def test_validation_reads_the_statistic_that_recorded_steps_wrote():
    """A state that ``call`` assigns under ``mixed_bfloat16``: replays of the recorded step write it without any version counter moving."""
    import keras_b200 as keras

    class Scaled(keras.layers.Layer):
        def build(self, shape):
            self.seen = self.add_weight(shape=(), initializer="zeros", trainable=False, name="seen")

        def call(self, t, training=False):
            if training:
                self.seen.assign_add(keras.ops.ones((), dtype="float32"))
            return t + keras.ops.cast(self.seen, t.dtype)

    def fitted(jit):
        keras.utils.set_random_seed(7)
        old = keras.config.dtype_policy()
        keras.config.set_dtype_policy("mixed_bfloat16")
        try:
            x = keras.Input((64,))
            m = keras.Model(x, keras.layers.Dense(8)(Scaled()(x)))
        finally:
            keras.config.set_dtype_policy(old)
        m.compile(keras.optimizers.SGD(0.0), "mse", jit_compile=jit)
        seen = []
        for _ in range(3):
            for _ in range(5):
                m.train_on_batch(data, target)
            with torch.no_grad():
                seen += [m(data, training=False).float() for _ in range(4)]
        return seen

    gc.collect()
    data, target = torch.randn(32, 64, device="cuda"), torch.zeros(32, 8, device="cuda")
    for a, b in zip(fitted("auto"), fitted(False)):
        assert torch.equal(a, b)


def test_inference_of_a_recorded_model_and_under_inference_mode():
    import keras_b200 as keras

    keras.utils.set_random_seed(1)
    model = _bf16_model(301)
    x = torch.randn(8, 16, 64, device="cuda")
    with torch.no_grad():
        for _ in range(3):
            model(x, training=False)
        gc.collect()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = model(x, training=False)
        for layer in model.layers[1:]:
            layer.kernel.value.mul_(-1.5)
        graph.replay()
        assert torch.allclose(out.float(), _plain(model, x).float(), atol=0.05, rtol=0.02)
    with torch.inference_mode():
        assert _agrees(model, x)
        built_inside = _bf16_model(301)
        assert all(_agrees(built_inside, x) for _ in range(3))
    assert all(_agrees(built_inside, x) for _ in range(3))
    loss = model(x, training=True).float().square().mean()
    loss.backward()
    assert all(v.value.grad is not None for v in model.trainable_variables)


def test_inference_leaves_nothing_behind():
    """Neither memory nor anything that keeps a variable from being copied or pickled."""
    import copy
    import pickle

    model = _bf16_model(301, 512)
    x = torch.randn(1, 16, 512, device="cuda")
    with torch.no_grad():
        model(x, training=False)
        held = torch.cuda.memory_allocated()
        for _ in range(3):
            model(x, training=False)
    assert torch.cuda.memory_allocated() == held
    kernel = model.layers[2].kernel
    for twin in (copy.deepcopy(kernel), pickle.loads(pickle.dumps(kernel))):
        assert torch.equal(twin.value.cpu(), kernel.value.cpu())


def test_inference_on_two_streams():
    import keras_b200 as keras

    keras.utils.set_random_seed(2)
    model = _bf16_model(301)
    x = torch.randn(8, 16, 64, device="cuda")
    side = torch.cuda.Stream()
    with torch.no_grad():
        want = _plain(model, x).float()
        side.wait_stream(torch.cuda.current_stream())
        for _ in range(2):
            with torch.cuda.stream(side):
                there = model(x, training=False)
        here = model(x, training=False)
        torch.cuda.synchronize()
        for out in (there, here):
            assert torch.allclose(out.float(), want, atol=0.05, rtol=0.02)


@pytest.mark.parametrize("K", [3, 5, 7])
@pytest.mark.parametrize("S", [1, 2])
@pytest.mark.parametrize("padding", ["same", "valid"])
@pytest.mark.parametrize("N,H,W,C", [(1, 7, 7, 8), (3, 9, 14, 40), (2, 15, 10, 144), (5, 8, 33, 264), (2, 29, 28, 320)])
def test_depthwise_convolution_and_gradients_against_64_bits(K, S, padding, N, H, W, C):
    from keras_b200.kernels import depthwise as dw

    g = torch.Generator(device="cuda").manual_seed(H * W + K)
    x = torch.randn((N, H, W, C), generator=g, device="cuda").bfloat16().requires_grad_(True)
    w = (torch.randn((K, K, C, 1), generator=g, device="cuda") / K).bfloat16().requires_grad_(True)
    y = dw.depthwise(x * 1, w, (S, S), padding, "channels_last", (1, 1))
    geometry = y.grad_fn.g
    xe, we = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    want = dw._composed(xe, we, geometry)
    assert y.shape == want.shape
    dy = torch.randn(y.shape, generator=g, device="cuda").bfloat16()
    y.backward(dy)
    want.backward(dy.double())
    rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()  # noqa: E731
    # one rounding to bf16 each (2^-9); the weight gradient sums N*OH*OW products in fp32 first
    assert rel(y, want) < 2.0 ** -8 and rel(x.grad, xe.grad) < 2.0 ** -8 and rel(w.grad, we.grad) < 2.0 ** -8


@pytest.mark.parametrize("K,S,N,H,C", [(3, 1, 64, 28, 192), (3, 2, 32, 57, 144), (5, 1, 16, 28, 8), (7, 2, 8, 30, 520), (3, 1, 40, 28, 64)])
def test_depthwise_weight_gradient_repeats_and_adds(K, S, N, H, C):
    from keras_b200.kernels import depthwise as dw

    g = torch.Generator(device="cuda").manual_seed(C)
    OH = -(-H // S)
    geometry = (N, H, H, C, OH, OH, K, S) + (max((OH - 1) * S + K - H, 0) // 2,) * 2
    x, dy = (torch.randn((N, n, n, C), generator=g, device="cuda").bfloat16() for n in (H, OH))
    first, again = (torch.full((K, K, C, 1), float("nan"), device="cuda") for _ in range(2))
    dw._launch(2, x, None, None, dy, first, geometry, accumulate=False)
    for _ in range(8):
        dw._launch(2, x, None, None, dy, again, geometry, accumulate=False)
        assert torch.equal(first, again)
    total = torch.ones((K, K, C, 1), device="cuda")
    dw._launch(2, x, None, None, dy, total, geometry)
    assert torch.equal(total, first + 1)
    w = torch.zeros((K, K, C, 1), dtype=torch.double, device="cuda", requires_grad=True)
    dw._composed(x.double(), w, geometry).backward(dy.double())
    # sums of N * OH * OW products in fp32
    assert ((first.double() - w.grad).norm() / w.grad.norm()).item() < 1e-5


def test_depthwise_routes():
    import keras_b200 as keras
    from keras_b200.kernels import depthwise as dw

    x = torch.randn(2, 9, 9, 16, device="cuda").bfloat16()
    w = torch.randn(3, 3, 16, 1, device="cuda").bfloat16()
    assert dw.depthwise(x, w, (1, 1), "same", "channels_first", (1, 1)) is None
    assert dw.depthwise(x, w, (1, 2), "same", "channels_last", (1, 1)) is None
    assert dw.depthwise(x, w, (1, 1), "same", "channels_last", (2, 2)) is None
    assert dw.depthwise(x, w.expand(3, 3, 16, 2).contiguous(), (1, 1), "same", "channels_last", (1, 1)) is None
    assert dw.depthwise(x.float(), w.float(), (1, 1), "same", "channels_last", (1, 1)) is None
    assert dw.depthwise(x[:, :2], w, (1, 1), "valid", "channels_last", (1, 1)) is None
    assert dw.depthwise(x, w, (1, 1), "same", "channels_last", (1, 1)) is None and dw.depthwise(x, w, (2, 2), "same", "channels_last", (1, 1)) is not None
    odd = torch.randn(2 * 9 * 9 * 16 + 1, device="cuda").bfloat16()[1:].reshape(2, 9, 9, 16)  # not 16-byte aligned
    flipped = x.transpose(1, 2)
    for t in (odd, flipped, x[:, ::2]):
        y = keras.ops.depthwise_conv(t, w, strides=2, padding="same", data_format="channels_last")
        want = keras.ops.depthwise_conv(t.float(), w.float(), strides=2, padding="same", data_format="channels_last")
        assert ((y.float() - want).norm() / want.norm()).item() < 2.0 ** -8
    # second derivatives
    xg = x.clone().requires_grad_(True)
    y = dw.depthwise(xg * 1, w, (1, 1), "same", "channels_last", (1, 1))
    (g,) = torch.autograd.grad((y.float() ** 2).sum(), xg, create_graph=True)
    assert torch.autograd.grad(g.float().square().sum(), xg)[0].isfinite().all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,C", [(5, 8), (4097, 48), (30000, 144)])
def test_batch_norm_with_relu6_is_the_two_layers(rows, C, dtype):
    from keras_b200.kernels import ops as kops

    torch.manual_seed(C)
    x = (torch.randn(rows, C, device="cuda") * 2).to(dtype).requires_grad_(True)
    gamma = (torch.rand(C, device="cuda") * 4 + 0.5).requires_grad_(True)
    beta = (torch.randn(C, device="cuda") + 1.5).requires_grad_(True)
    dy = torch.randn(rows, C, device="cuda").to(dtype)
    results = []
    for fused in (True, False):
        mm, mv = torch.zeros(C, device="cuda"), torch.ones(C, device="cuda")
        args = (x, gamma, beta, None, mm, mv, 0.9, 1e-3)
        y = kops.FusedBatchNormAct.apply(*args, True, None, None, None, 6.0) if fused else torch.nn.functional.relu6(kops.FusedBatchNormAct.apply(*args, False))
        results.append((y.detach(),) + torch.autograd.grad(y, (x, gamma, beta), dy))
    # the statistics are fp32 atomic sums (a few 2^-24 apart from run to run), the output is rounded once
    step = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-5
    (y0, dx0, dg0, db0), (y1, dx1, dg1, db1) = results
    assert torch.allclose(y0.float(), y1.float(), rtol=step, atol=step)
    # an element that those sums move across a bound gains or loses its gradient: hardly any may
    assert (~torch.isclose(dx0.float(), dx1.float(), rtol=4 * step, atol=4 * step * dx1.float().abs().max().item())).float().mean().item() < 1e-3
    for a, b in ((dg0, dg1), (db0, db1)):
        assert torch.allclose(a, b, rtol=1e-2, atol=1e-2 * b.abs().max().item())


def test_model_with_relu6_folds_it_into_the_normalisation():
    import keras_b200 as keras

    L = keras.layers
    keras.utils.set_random_seed(3)
    x = keras.Input((8, 8, 16))
    h = L.ReLU(6.0)(L.BatchNormalization()(L.Conv2D(32, 1)(x)))
    h = L.Activation("relu6")(L.BatchNormalization()(L.DepthwiseConv2D(3, padding="same")(h)))
    model = keras.Model(x, L.ReLU(4.0)(L.BatchNormalization()(L.Conv2D(16, 1)(h))))
    data = torch.randn(4, 8, 8, 16, device="cuda") * 3
    for training in (False, True):
        state = [v.value.clone() for v in model.weights]
        got = model(data, training=training)
        for v, s in zip(model.weights, state):
            v.assign(s)
        want = data
        for layer in model.layers[1:]:
            want = layer(want, training=training)
        for v, s in zip(model.weights, state):
            v.assign(s)
        assert torch.allclose(got, want, atol=1e-4, rtol=1e-4)
    from keras_b200.models import fusion

    plan = fusion.build_plan(model)
    assert list(plan.values()).count("consume_relu") == 2  # the bound of four keeps its own layer


@pytest.mark.parametrize("rows,C", [(64, 16), (4096, 1024), (20011, 144)])  # registers, the ring of bulk copies, both at no power of two
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind", ["relu", "relu6", "relu + residual"])
def test_batch_norm_with_a_rectifier_keeps_nan(rows, C, dtype, kind):
    """A channel whose statistics are no numbers stays so, values and gradients, as the layers one by one have it."""
    from keras_b200.kernels import ops as kops

    g = torch.Generator(device="cuda").manual_seed(C)
    x = torch.randn((rows, C), generator=g, device="cuda").to(dtype)
    x[3, 5], x[4, 6], x[5, 7] = float("nan"), float("inf"), 3.0
    res = torch.randn((rows, C), generator=g, device="cuda").to(dtype).requires_grad_(True) if "residual" in kind else None
    if res is not None:
        with torch.no_grad():
            res[7, 9] = float("nan")
    x.requires_grad_(True)
    gamma, beta = torch.ones(C, device="cuda", requires_grad=True), torch.zeros(C, device="cuda", requires_grad=True)
    mean, var = torch.zeros(C, device="cuda"), torch.ones(C, device="cuda")
    y = kops.FusedBatchNormAct.apply(x, gamma, beta, res, mean, var, 0.9, 1e-3, True, None, None, None, 6.0 if kind == "relu6" else None)
    bad = torch.zeros((rows, C), dtype=torch.bool, device="cuda")
    bad[:, 5:7] = True
    grad_bad = bad.clone()
    if res is not None:
        bad[7, 9] = True
    assert torch.equal(y.isnan(), bad)
    assert torch.equal(mean.isfinite(), ~bad[0]) and torch.equal(var.isnan(), bad[0])
    y.backward(torch.ones_like(y))
    assert torch.equal(x.grad.isnan(), grad_bad)
    if res is not None:
        assert res.grad[7, 9].item() == 1.0  # the gradient passes where the sum is no number
    scale = torch.ones(C, device="cuda")
    scale[5] = float("nan")
    out = kops.bn_inference(x.detach(), scale, beta.detach(), None, True, 6.0 if kind == "relu6" else None)
    assert out[:, 5].isnan().all() and out[3, 5].isnan() and not out[:, 8].isnan().any()


def _odd_chains():
    """Chains in which one layer is more than the fused kernel that could stand for its neighbours: ``{name: (input shape, build)}``."""
    import keras_b200 as keras

    L = keras.layers

    def relu(t):
        return t * 0 + 7

    def linear(t):
        return t * 0 + 2

    class Rectifier(L.ReLU):
        def call(self, t):
            return t * 0 + 5

    class Norm(L.BatchNormalization):
        def call(self, t, training=None, mask=None):
            return t * 0 - 3

    class Sum(L.Add):
        def _merge_function(self, inputs):
            return inputs[0] * 0 + 4

    class Conv(L.Conv2D):
        def call(self, t):
            return t * 0 + 9

    class Frame(L.ZeroPadding2D):
        def call(self, t):
            return torch.nn.functional.pad(t, (0, 0, 1, 1, 1, 1), value=100.0)

    conv = lambda t, **k: L.Conv2D(16, 1, **k)(t)  # noqa: E731
    norm = lambda t, **k: L.BatchNormalization(**k)(t)  # noqa: E731
    image = (8, 8, 16)
    return {
        "relu6 in float32": (image, lambda x: L.ReLU(6.0, dtype="float32")(norm(conv(x)))),
        "relu in float32": (image, lambda x: L.ReLU(dtype="float32")(norm(conv(x)))),
        "norm in float32": (image, lambda x: L.ReLU(6.0)(norm(conv(x), dtype="float32"))),
        "sum in float32": (image, lambda x: L.ReLU()(L.Add(dtype="float32")([norm(conv(x)), x]))),
        "rectified sum in float32": (image, lambda x: L.ReLU(dtype="float32")(L.Add()([norm(conv(x)), x]))),
        "relu6 with a penalty": (image, lambda x: L.ReLU(6.0, activity_regularizer="l2")(norm(conv(x)))),
        "relu with a penalty": (image, lambda x: L.ReLU(activity_regularizer="l2")(norm(conv(x)))),
        "norm with a penalty": (image, lambda x: L.ReLU()(norm(conv(x), activity_regularizer="l2"))),
        "sum with a penalty": (image, lambda x: L.Add(activity_regularizer="l2")([norm(conv(x)), x])),
        "relu6 of one's own": (image, lambda x: Rectifier(6.0)(norm(conv(x)))),
        "relu of one's own": (image, lambda x: Rectifier()(norm(conv(x)))),
        "function called relu": (image, lambda x: L.Activation(relu)(norm(conv(x)))),
        "convolution with a function called linear": (image, lambda x: L.ReLU()(norm(conv(x, activation=linear)))),
        "norm of one's own": (image, lambda x: L.ReLU(6.0)(Norm()(conv(x)))),
        "sum of one's own": (image, lambda x: Sum()([norm(conv(x)), x])),
        "convolution of one's own": (image, lambda x: L.ReLU(6.0)(norm(Conv(16, 1)(x)))),
        "padding of one's own": (image, lambda x: L.MaxPooling2D(3, 2)(Frame(1)(x))),
        "frozen norm": (image, lambda x: L.ReLU(6.0)(L.BatchNormalization()(x, training=False))),
        "masked norm": ((6, 8), lambda x: L.ReLU(6.0)(norm(L.Masking()(x)))),
    }


@pytest.mark.parametrize("policy", ["float32", "mixed_bfloat16"])
@pytest.mark.parametrize("training", [False, True])
def test_folded_chains_answer_as_their_layers_do(policy, training):
    """Results, their type, penalties and masks of a whole model against its layers called one by one."""
    import keras_b200 as keras

    old = keras.config.dtype_policy()
    for name, (shape, build) in _odd_chains().items():
        keras.utils.set_random_seed(5)
        keras.config.set_dtype_policy(policy)
        try:
            x = keras.Input(shape)
            model = keras.Model(x, build(x))
        finally:
            keras.config.set_dtype_policy(old)
        data = torch.randn((4,) + shape, device="cuda") * 2
        data[:, 3:] = data[:, 3:] * (len(shape) == 3)  # positions of a sequence that are masked
        state = [v.value.clone() for v in model.weights]
        with torch.no_grad():
            got = model(data, training=training)
            penalties = len(model.losses)
            after = [v.value.clone() for v in model.weights]
            for v, s in zip(model.weights, state):
                v.assign(s)
            env = {id(t): data for t in model.inputs}
            for node in model._ordered_nodes():
                if node.input_tensors:
                    args, kwargs = node.arguments.fill_in(env)
                    if not isinstance(node.operation, keras.layers.BatchNormalization) or "training" in kwargs:
                        env[id(node.outputs[0])] = node.operation(*args, **kwargs)
                    else:
                        env[id(node.outputs[0])] = node.operation(*args, training=training)
        want = env[id(model.outputs[0])]
        assert got.dtype == want.dtype == keras.ops.zeros((), dtype=model.outputs[0].dtype).dtype, name
        assert (getattr(got, "_keras_mask", None) is None) == (getattr(want, "_keras_mask", None) is None), name
        assert penalties == sum(layer.activity_regularizer is not None for layer in model.layers), name
        # a fused chain keeps float32 between its parts where layers of their own round to the compute type
        step = 2.0 ** -6 if policy != "float32" else 1e-4
        assert torch.allclose(got.float(), want.float(), rtol=step, atol=step), name
        for a, v in zip(after, model.weights):
            assert torch.allclose(a, v.value, rtol=step, atol=step), name


@pytest.mark.parametrize("rows", [(8, 1), (1, 8)])
@pytest.mark.parametrize("training", [False, True])
def test_a_sum_behind_a_norm_broadcasts(rows, training):
    """Two inputs of declared equal shapes and different batches: the kernel's element by element sum would read behind the smaller one."""
    import keras_b200 as keras

    L = keras.layers
    a, b = keras.Input((6, 6, 16)), keras.Input((6, 6, 16))
    model = keras.Model([a, b], L.ReLU()(L.Add()([L.BatchNormalization()(L.Conv2D(16, 1)(a)), b])))
    xa, xb = (torch.randn((n, 6, 6, 16), device="cuda") for n in rows)
    conv, norm = (next(layer for layer in model.layers if isinstance(layer, t)) for t in (L.Conv2D, L.BatchNormalization))
    state = [v.value.clone() for v in norm.weights]
    with torch.no_grad():
        got = model([xa, xb], training=training)
        for v, s in zip(norm.weights, state):
            v.assign(s)
        want = torch.relu(norm(conv(xa), training=training) + xb)
    assert got.shape == want.shape and torch.allclose(got, want, atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("relu,res", [(True, True), (True, False), (False, False)])
@pytest.mark.parametrize("rows,C", [(20011, 144), (15003, 192), (70001, 48), (3001, 960), (9001, 320), (2200, 1000), (600, 4096), (30, 24)])
def test_batch_norm_at_channel_counts_that_are_no_power_of_two(rows, C, relu, res):
    """The bulk-copy ring and the register kernels, with ragged last tiles; against the same mathematics in 64 bits."""
    from keras_b200.kernels import ops as kops

    torch.manual_seed(C)
    x = (torch.randn(rows, C, device="cuda") * 1.5 + 0.25).bfloat16().requires_grad_(True)
    r = torch.randn(rows, C, device="cuda").bfloat16().requires_grad_(True) if res else None
    gamma, beta = (torch.rand(C, device="cuda") + 0.5).requires_grad_(True), torch.randn(C, device="cuda").requires_grad_(True)
    mm, mv = torch.zeros(C, device="cuda"), torch.ones(C, device="cuda")
    y = kops.FusedBatchNormAct.apply(x, gamma, beta, r, mm, mv, 0.9, 1e-3, relu)
    dy = torch.randn_like(y)
    got = torch.autograd.grad(y, [x, gamma, beta] + ([r] if res else []), dy)
    kops.check_stream_kernels()
    xe, ge, be = (t.detach().double().requires_grad_(True) for t in (x, gamma, beta))
    re = r.detach().double().requires_grad_(True) if res else None
    mean, var = xe.mean(0), xe.var(0, correction=0)
    ref = (xe - mean) * torch.rsqrt(var + 1e-3) * ge + be + (re if res else 0)
    # the mask that the kernel took: a value within rounding of zero may go either way
    ref = ref * (y.double() > 0) if relu else ref
    want = torch.autograd.grad(ref, [xe, ge, be] + ([re] if res else []), dy.double())
    rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()  # noqa: E731
    assert rel(y, ref) < 2.0 ** -8
    for a, b, bound in zip(got, want, (2.0 ** -8, 2.0 ** -10, 2.0 ** -10, 2.0 ** -8)):  # dx and dres rounded to bf16; sums in fp32 of exact products
        assert rel(a, b) < bound


@pytest.mark.parametrize("M,K,N", [(77, 64, 301), (129, 72, 136), (1001, 256, 512), (8446, 128, 1001), (2667, 512, 2048), (3, 768, 5001), (8193, 32, 21), (20000, 384, 37)])
def test_dense_products_at_any_number_of_rows(M, K, N):
    from keras_b200.kernels import gemm

    torch.manual_seed(M)
    x = torch.randn(M, K, device="cuda").bfloat16().requires_grad_(True)
    w = (torch.randn(K, N, device="cuda") * K ** -0.5).bfloat16().requires_grad_(True)
    b = torch.randn(N, device="cuda").requires_grad_(True)
    assert gemm._qualifies(x, w) == (2 * M * N * K >= gemm._MIN_WORK)
    y = gemm.GemmFn.apply(x, w, b, None, None)
    dy = torch.randn(M, N, device="cuda").bfloat16()
    y.backward(dy)
    gemm.check_errors()
    xe, we, be = (t.detach().double().requires_grad_(True) for t in (x, w, b))
    ye = xe @ we + be
    ye.backward(dy.double())
    rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()  # noqa: E731
    assert rel(y, ye) < 2.0 ** -8 and rel(x.grad, xe.grad) < 2.0 ** -8 and rel(w.grad, we.grad) < 2.0 ** -8 and rel(b.grad, be.grad) < 1e-5
    with torch.no_grad():  # the fused form of inference
        out, done = gemm.dense(x, w, b, "gelu") or (None, None)
        if out is not None:
            assert done and rel(out, torch.nn.functional.gelu(ye)) < 2.0 ** -8


def test_shortcut_and_branch_share_the_cast_of_a_float32_input():
    import keras_b200 as keras

    L = keras.layers
    old = keras.config.dtype_policy()
    keras.config.set_dtype_policy("mixed_bfloat16")
    try:
        x = keras.Input((16, 16, 64))
        a = L.BatchNormalization()(L.Conv2D(64, 1, use_bias=False)(x))
        b = L.BatchNormalization()(L.Conv2D(64, 1, use_bias=False)(x))
        model = keras.Model(x, L.ReLU()(L.Add()([a, b])))
    finally:
        keras.config.set_dtype_policy(old)
    data = torch.randn(64, 16, 16, 64, device="cuda")
    from keras_b200.models import fusion

    casts = {}
    convs = [layer for layer in model.layers if isinstance(layer, L.Conv2D)]
    first, second = (fusion.shared_cast(layer, data, casts) for layer in convs)
    assert first is second and first.dtype == torch.bfloat16 and len(casts) == 1
    assert fusion.shared_cast(convs[0], data.clone(), casts) is not first
    out = model(data, training=True)
    assert out.dtype == torch.bfloat16 and torch.isfinite(out).all()
    grown = data.clone().requires_grad_(True)  # with a gradient the casts stay apart: their gradients are summed in float32
    model(grown, training=True).float().square().mean().backward()
    assert grown.grad is not None and grown.grad.dtype == torch.float32


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 9), (64, 301), (7, 2047), (70000, 5), (768, 50257)])
def test_padded_matrices(rows, cols):
    from keras_b200.kernels import ops as kops

    torch.manual_seed(cols)
    w = torch.randn(rows, cols, device="cuda").bfloat16()
    wide = -(-cols // 8) * 8
    padded = kops.pad_columns(w, wide)
    assert torch.equal(padded, torch.nn.functional.pad(w, (0, wide - cols)))
    odd = torch.randn(rows * cols + 1, device="cuda").bfloat16()[1:].reshape(rows, cols)  # not even 4-byte aligned
    assert torch.equal(kops.pad_columns(odd, wide + 8)[:, :cols], odd)
    total = torch.randn(rows, cols, device="cuda")
    want = total + padded[:, :cols].float()
    assert torch.equal(kops.add_rows(total, padded[:, :cols]), want)
    assert torch.equal(kops.add_rows(total, w), want + w.float())


@pytest.mark.parametrize("activation", ["relu", "silu", "gelu"])
@pytest.mark.parametrize("rows,width,use_bias", [((3, 5), 64, True), ((1000,), 264, True), ((5000,), 512, False), ((77, 260), 1024, True), ((20100,), 512, True)])
def test_dense_with_an_activation_and_its_gradient(activation, rows, width, use_bias):
    import keras_b200 as keras

    old = keras.config.dtype_policy()
    keras.config.set_dtype_policy("mixed_bfloat16")
    try:
        layer = keras.layers.Dense(width, activation=activation, use_bias=use_bias)
        plain = keras.layers.Dense(width, use_bias=use_bias)
    finally:
        keras.config.set_dtype_policy(old)
    torch.manual_seed(width)
    x = torch.randn(rows + (256,), device="cuda").bfloat16().requires_grad_(True)
    dy = torch.randn(rows + (width,), device="cuda").bfloat16()
    layer(x), plain(x)
    for a, b in zip(plain.weights, layer.weights):
        a.assign(b.value + 0.1 * torch.randn(tuple(b.shape), device="cuda"))
        b.assign(a.value)
    results = []
    for run in (layer, lambda t: getattr(torch.nn.functional, activation)(plain(t))):
        y = run(x)
        which = layer if run is layer else plain
        results.append([y.detach()] + list(torch.autograd.grad(y, [x] + [v.value for v in which.trainable_variables], dy)))
    for a, b in zip(*results):
        # the same rounded value ahead of the activation; each result is rounded once more
        assert ((a.float() - b.float()).norm() / b.float().norm()).item() < 2.0 ** -8


@pytest.mark.parametrize("rows,width", [(1000, 256), (1001, 256), (1001, 301)])
@pytest.mark.parametrize("activation", [None, "gelu", "silu"])
def test_second_derivatives_of_a_dense_layer(rows, width, activation):
    """A penalty on the gradient of the input: it reaches the weights, at every route of the product."""
    import keras_b200 as keras

    old = keras.config.dtype_policy()
    keras.config.set_dtype_policy("mixed_bfloat16")
    try:
        layer = keras.layers.Dense(width, activation=activation)
    finally:
        keras.config.set_dtype_policy(old)
    torch.manual_seed(rows + width)
    x = torch.randn(rows, 256, device="cuda").bfloat16().requires_grad_(True)
    layer(x)
    layer.bias.assign(torch.randn(width, device="cuda") * 0.3)
    y = layer(x)
    (g,) = torch.autograd.grad(y.float().square().sum(), x, create_graph=True)
    got = torch.autograd.grad(g.float().square().sum(), [layer.kernel.value, layer.bias.value])
    xe, w, b = (t.detach().double().requires_grad_(True) for t in (x, layer.kernel.value, layer.bias.value))
    ye = torch.matmul(xe, w) + b
    ye = ye if activation is None else getattr(torch.nn.functional, activation)(ye)
    (ge,) = torch.autograd.grad(ye.square().sum(), xe, create_graph=True)
    want = torch.autograd.grad(ge.square().sum(), [w, b])
    assert ((g.double() - ge).norm() / ge.norm()).item() < 2.0 ** -6
    for a, e in zip(got, want):  # a chain of some eight roundings to bf16
        assert ((a.double() - e).norm() / e.norm()).item() < 2.0 ** -6


@pytest.mark.parametrize("rows,N", [(1001, 301), (2048, 297), (1001, 303)])
def test_gradient_of_padded_columns_leaves_its_neighbours_alone(rows, N):
    """A product of odd width beside other columns: its gradient is a view of the whole gradient, with the same pitch as the padded one."""
    from keras_b200.kernels import gemm

    g = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn((rows, 256), generator=g, device="cuda").bfloat16().requires_grad_(True)
    w = torch.randn((256, N), generator=g, device="cuda").bfloat16().requires_grad_(True)
    b = torch.randn(N, generator=g, device="cuda").requires_grad_(True)
    other = torch.randn((rows, -N % 8), generator=g, device="cuda").bfloat16().requires_grad_(True)
    coef = torch.randn((rows, N - N % 8 + 8), generator=g, device="cuda").bfloat16()
    coef[0, N:] = float("inf")
    kept = coef.clone()
    y = torch.cat([gemm.GemmFn.apply(x, w, b), other], dim=1)
    y.backward(coef)
    gemm.check_errors()
    assert torch.equal(coef, kept) and torch.equal(other.grad, kept[:, N:])
    d = kept[:, :N].double()
    for got, want in ((x.grad, d @ w.detach().double().t()), (w.grad, x.detach().double().t() @ d), (b.grad, d.sum(0))):
        assert ((got.double() - want).norm() / want.norm()).item() < 2.0 ** -8


def _transformed_models():
    import keras_b200 as keras

    L = keras.layers
    old = keras.config.dtype_policy()
    try:
        keras.config.set_dtype_policy("mixed_bfloat16")
        for rows in (1000, 1001):
            for activation in (None, "relu", "gelu"):
                x = keras.Input((rows, 256))
                yield f"dense {rows} {activation}", keras.Model(x, L.Dense(256, activation=activation)(x)), (1, rows, 256)
        x = keras.Input((40, 256))
        yield "attention", keras.Model(x, L.MultiHeadAttention(4, 64)(x, x)), (2, 40, 256)
        yield "depthwise", keras.Sequential([keras.Input((12, 12, 16)), L.DepthwiseConv2D(3, strides=2), L.BatchNormalization(), L.ReLU(6.0)]), (2, 12, 12, 16)
        keras.config.set_dtype_policy("float32")
        yield "lstm", keras.Sequential([keras.Input((5, 8)), L.LSTM(32)]), (3, 5, 8)
        x = keras.Input((8, 8, 16))
        yield "chain", keras.Model(x, L.ReLU(6.0)(L.BatchNormalization()(L.Conv2D(16, 3, padding="same")(x)))), (2, 8, 8, 16)
    finally:
        keras.config.set_dtype_policy(old)


@pytest.mark.parametrize("recording", [False, True])
def test_forward_mode_and_function_transforms_see_every_layer(recording):
    """A tangent against the reverse mode (<J t, J t> = <t, J' J t>), and a mapped call against a single one: with and without gradients."""
    import keras_b200 as keras
    from torch.autograd import forward_ad

    keras.utils.set_random_seed(4)
    for name, model, shape in _transformed_models():
        g = torch.Generator(device="cuda").manual_seed(2)
        x, t = (torch.randn(shape, generator=g, device="cuda") for _ in range(2))
        with torch.set_grad_enabled(recording):
            plain = model(x, training=False)
            with torch.nn.attention.sdpa_kernel(torch.nn.attention.SDPBackend.MATH):  # the one library attention with these derivatives
                with forward_ad.dual_level():
                    tangent = forward_ad.unpack_dual(model(forward_ad.make_dual(x, t), training=False)).tangent
                also = keras.ops.jvp(lambda a: model(a, training=False), (x,), (t,))[1]
                many = torch.func.vmap(lambda a: model(a, training=False))(torch.stack([x, x + t]))
        assert tangent is not None, name
        xg = x.clone().requires_grad_(True)
        (back,) = torch.autograd.grad(model(xg, training=False), xg, tangent.detach())
        want = (back * t).sum().item()
        for got in (tangent, also):  # sums over thousands of products of bf16 numbers
            assert got.detach().float().square().sum().item() == pytest.approx(want, rel=0.02 if plain.dtype == torch.bfloat16 else 1e-3), name
        assert torch.allclose(many[0].float(), plain.float(), atol=0.03, rtol=0.03), name


@pytest.mark.parametrize("act,fn", [(1, torch.relu), (3, torch.nn.functional.silu), (4, torch.nn.functional.gelu)])
def test_activation_derivatives_at_infinities_and_nan(act, fn):
    from keras_b200.kernels import ops as kops

    values = [float("inf"), float("-inf"), float("nan"), 0.0, -0.0, 1.5, -1.5, 300.0, -300.0, 3e38, -3e38]
    pairs = torch.cartesian_prod(torch.tensor(values), torch.tensor(values)).cuda().bfloat16()
    dy, z = (torch.nn.functional.pad(c, (0, 128 - len(c))).reshape(8, 16).contiguous() for c in pairs.t())
    z = z.requires_grad_(True)
    (want,) = torch.autograd.grad(fn(z), z, dy)
    got = kops.activation_backward(dy, z.detach(), act)[0]
    same = (got == want) | (got.isnan() & want.isnan()) | ((got.float() - want.float()).abs() <= 2.0 ** -8 * want.float().abs() + 1e-30)
    assert same.all(), torch.stack([dy[~same], z[~same], got[~same], want[~same]], 1)


@pytest.mark.parametrize("rows", [8, 1001, 5000])
def test_dense_with_a_relu_keeps_nan_in_inference(rows):
    import keras_b200 as keras

    layer = keras.layers.Dense(256, activation="relu", dtype="bfloat16")
    x = torch.randn(rows, 512, device="cuda").bfloat16()
    x[5, 7] = float("nan")
    with torch.no_grad():
        out = layer(x)
    assert out[5].isnan().all() and not out[:5].isnan().any() and not out[6:].isnan().any() and (out[:5] >= 0).all()


def test_a_function_of_the_users_own_is_not_taken_for_a_known_activation():
    import keras_b200 as keras

    def gelu(x):
        return x * 3.0

    old = keras.config.dtype_policy()
    keras.config.set_dtype_policy("mixed_bfloat16")
    try:
        layer = keras.layers.Dense(256, activation=gelu)
    finally:
        keras.config.set_dtype_policy(old)
    x = torch.randn(256, 256, device="cuda").bfloat16()
    for grad in (True, False):
        with torch.set_grad_enabled(grad):
            y, want = layer(x), 3.0 * torch.matmul(x.float(), layer.kernel.value.float())
            assert ((y.float() - want).norm() / want.norm()).item() < 2.0 ** -7


def test_a_quantised_layer_calls_the_function_it_was_given():
    import keras_b200 as keras

    def gelu(x):
        return x * 0 + 3.0

    x = torch.randn(128, 64, device="cuda")
    for layer in (keras.layers.Dense(64, activation=gelu), keras.layers.EinsumDense("ab,bc->ac", output_shape=64, bias_axes="c", activation=gelu)):
        layer(x)
        layer.quantize("int8")
        with torch.no_grad():
            assert torch.equal(layer(x), torch.full((128, 64), 3.0, device="cuda"))
    for name in ("relu", "gelu", "silu"):
        layer = keras.layers.Dense(64, activation=name)
        layer(x)
        layer.quantize("int8")
        with torch.no_grad():
            out = layer(x)
            layer.activation = keras.activations.linear
            want = getattr(torch.nn.functional, name)(layer(x))
        assert torch.allclose(out, want, atol=1e-5, rtol=1e-5)


def test_exact_gelu_of_the_epilogue_and_its_derivative_over_the_whole_range():
    from keras_b200.kernels import gemm, ops as kops

    # the product with the identity hands every value of x to the epilogue as it is
    x = torch.cat([torch.linspace(-14, 14, 64 * 1000 - 64), torch.tensor([0.0, -0.0, 1e-30, -1e-30] * 8 + [30.0, -30.0, 1e4, -1e4] * 8)]).reshape(1000, 64).cuda().bfloat16()
    eye = torch.eye(64, device="cuda").bfloat16()
    xe = x.double()
    cdf = 0.5 * torch.special.erfc(-xe * 0.5 ** 0.5)  # 1 + erf cancels for negative values, in 64 bits too
    want, slope = xe * cdf, cdf + xe * torch.exp(-0.5 * xe * xe) * 0.3989422804014327
    out = gemm.gemm(x, eye, 0, 1, 1000, 64, 64, act=4, out_dtype=torch.float32)
    # float32: 2.5e-6 of the value (the exponent's rounding grows with x^2 beyond 6) and nothing below 1e-30
    assert torch.all((out.double() - want).abs() <= 2e-5 * want.abs() + 1e-30)
    small = x.abs() < 6
    assert torch.all((out.double() - want).abs()[small] <= 4e-6 * want.abs()[small] + 1e-30)
    one = torch.ones_like(x)
    dz, _ = kops.activation_backward(one, x, 4)
    assert torch.all((dz.double() - slope).abs() <= 2.0 ** -8 * slope.abs() + 2e-6)  # one rounding to bf16; the slope itself crosses zero
    nan = torch.full((8, 64), float("nan"), device="cuda").bfloat16()
    assert gemm.gemm(nan, eye, 0, 1, 8, 64, 64, act=4).isnan().all() and kops.activation_backward(one[:8].contiguous(), nan, 4)[0].isnan().all()


def test_gelu_into_float32_is_as_accurate_as_the_library():
    from keras_b200.kernels import gemm

    x = torch.cat([torch.linspace(-2, 2, 64 * 999), torch.linspace(-0.01, 0.01, 64)]).reshape(1000, 64).cuda().bfloat16()
    xe = x.double()
    want = xe * 0.5 * torch.special.erfc(-xe * 0.5 ** 0.5)
    out = gemm.gemm(x, torch.eye(64, device="cuda").bfloat16(), 0, 1, 1000, 64, 64, act=4, out_dtype=torch.float32).double()
    off = (out - want).abs() / want.abs().clamp_min(1e-30)
    # half an ulp (2^-24) each for the sum and two products, up to two ulps of erf; relative to 1 + erf, which is 0.317 at -1 and 0.0455 at -2
    for low, high, bound in ((0, 2, 5 * 2.0 ** -24), (-1, 0, 5 * 2.0 ** -24 / 0.317), (-2, -1, 5 * 2.0 ** -24 / 0.0455)):
        assert off[(x >= low) & (x <= high)].max().item() <= bound
    assert off[(x >= -1) & (x <= 1)].square().mean().sqrt().item() < 1e-7


def test_int8_operands_are_not_taken_for_those_of_a_freed_kernel():
    """Kernels that take one another's place in memory (unpacked int4 kernels of equal layers, a second model): each its own product."""
    from keras_b200.kernels import dispatch

    x = torch.randint(-127, 128, (64, 256), device="cuda", dtype=torch.int8)
    one = torch.ones((64, 1), device="cuda")
    seen = set()
    for seed in range(64):  # until memory has been reused, which is the allocator's to decide
        g = torch.Generator(device="cuda").manual_seed(seed)
        kernel = torch.randint(-127, 128, (256, 128), generator=g, device="cuda", dtype=torch.int8)
        scale = torch.rand(128, generator=g, device="cuda") + 0.5
        reused = kernel.data_ptr() in seen
        seen.add(kernel.data_ptr())
        for view in (kernel, kernel.reshape(256, 8, 16).reshape(256, -1), kernel):
            out = dispatch.int8_matmul(x, view, one, scale, out_dtype=torch.float32)
            want = (x.double() @ kernel.double()) / scale.double()
            assert torch.allclose(out.double(), want, rtol=1e-6, atol=1e-3)  # exact integer sums below 2^24, a reciprocal and a product rounded
        kernel.neg_()  # changed in place
        assert torch.allclose(dispatch.int8_matmul(x, kernel, one, scale, out_dtype=torch.float32).double(), -want, rtol=1e-6, atol=1e-3)
        if reused:
            return
        del kernel, view, scale
    raise AssertionError("no kernel took the place of another one")


def _anywhere(t):
    """The same values in a contiguous tensor that starts one element behind a 16-byte line."""
    return torch.cat([t.new_zeros(1), t.detach().reshape(-1)])[1:].reshape(t.shape)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_layers_take_tensors_and_gradients_that_start_anywhere(dtype):
    """The gradient of a concatenation of flattened tensors is contiguous and starts where the one before ends."""
    import keras_b200 as keras
    from keras_b200.kernels import ops as kops

    L = keras.layers
    name = "float32" if dtype == torch.float32 else "mixed_bfloat16"
    g = torch.Generator(device="cuda").manual_seed(3)
    ones, zeros = torch.ones(64, device="cuda"), torch.zeros(64, device="cuda")

    def norm(x, res=None, cap=None):
        return kops.FusedBatchNormAct.apply(x, ones, zeros, res, zeros.clone(), ones.clone(), 0.9, 1e-3, True, None, None, None, cap)

    calls = {"norm + relu": lambda x: norm(x), "norm + relu6": lambda x: norm(x, cap=6.0), "norm + sum": lambda x: norm(x, x)}
    layers = {"max": L.MaxPooling2D(2), "average": L.AveragePooling2D(2), "global": L.GlobalAveragePooling2D(), "conv": L.Conv2D(64, 3), "dense": L.Dense(128),
              "dense + gelu": L.Dense(128, activation="gelu"), "depthwise": L.DepthwiseConv2D(3, strides=2), "layer norm": L.LayerNormalization()}
    for key, layer in layers.items():
        layer.dtype_policy = keras.dtype_policies.get(name)
        calls[key] = layer
    for key, call in calls.items():
        x = torch.randn((4, 16, 16, 64), generator=g, device="cuda").to(dtype)
        results = []
        for place in (lambda t: t, _anywhere):
            xi = place(x).requires_grad_(True)
            assert place is not _anywhere or xi.data_ptr() % 16
            y = call(xi)
            dy = torch.randn(y.shape, generator=torch.Generator(device="cuda").manual_seed(4), device="cuda").to(y.dtype)
            (dx,) = torch.autograd.grad(y, xi, place(dy))
            results.append((y.detach(), dx))
        for a, b in zip(*results):
            assert ((a.float() - b.float()).norm() / a.float().norm()).item() < 2.0 ** -7, key  # an unaligned one may run in the library
    out = kops.bn_inference(_anywhere(x), ones, zeros, _anywhere(x), True)
    assert torch.equal(out, torch.relu(x.float() * 1 + x.float()).to(dtype))
    table, ids = torch.randn((33, 64), generator=g, device="cuda"), torch.randint(0, 33, (40,), generator=g, device="cuda")
    rows = kops.FusedEmbedding.apply(_anywhere(table).requires_grad_(True), ids, torch.float32, None)
    assert torch.equal(rows, table[ids])
    rows.backward(_anywhere(torch.ones_like(rows)))


def test_int8_operands_of_two_streams():
    """What is laid out for a kernel on one stream, behind other work, is not yet there for a second one."""
    from keras_b200.kernels import dispatch

    x = torch.randint(-127, 128, (64, 512), device="cuda", dtype=torch.int8)
    kernel = torch.randint(-127, 128, (512, 1024), device="cuda", dtype=torch.int8)
    one, scale = torch.ones((64, 1), device="cuda"), torch.rand(1024, device="cuda") + 0.5
    want = (x.double() @ kernel.double()) / scale.double()
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    dispatch.int8_matmul(x, kernel.clone(), one, scale.clone(), out_dtype=torch.float32)  # all kernels are loaded
    with torch.cuda.stream(first):
        torch.cuda._sleep(1)
        torch.full((1 << 22,), 77, device="cuda", dtype=torch.int8)  # leaves something else in the memory that is handed out next
    torch.cuda.synchronize()
    outs = []
    for stream in (first, second):
        with torch.cuda.stream(stream):
            if stream is first:
                torch.cuda._sleep(200_000_000)  # a tenth of a second
            outs.append(dispatch.int8_matmul(x, kernel, one, scale, out_dtype=torch.float32))
    torch.cuda.synchronize()
    for out in outs:
        assert torch.allclose(out.double(), want, rtol=1e-6, atol=1e-3)


@pytest.mark.parametrize("n", [8, 4096, 8 * 148 * 16 * 256 * 2 + 8, 999])
def test_copy_and_cast(n):
    from keras_b200.kernels import ops as kops

    src = torch.randn(n, device="cuda")
    src[:3] = torch.tensor([float("nan"), float("inf"), -3.4e38])
    dst, dst16 = torch.zeros_like(src), torch.zeros(n, device="cuda", dtype=torch.bfloat16)
    kops.copy_and_cast(src, dst, dst16)
    assert torch.equal(dst[1:], src[1:]) and dst[0].isnan() and torch.equal(dst16[1:], src[1:].to(torch.bfloat16)) and dst16[0].isnan()


def test_recorded_step_reads_the_rounded_batch_of_each_replay():
    """A float32 batch into convolutions, also read as it is: each replay answers as the eager step does, batch by batch."""
    import keras_b200 as keras

    def build():
        keras.utils.set_random_seed(3)
        keras.config.set_dtype_policy("mixed_bfloat16")
        try:
            x = keras.Input((16, 16, 64))
            a, b = (keras.layers.ReLU()(keras.layers.BatchNormalization()(keras.layers.Conv2D(64, k, padding="same", use_bias=False)(x))) for k in (1, 3))
        finally:
            keras.config.set_dtype_policy("float32")
        h = keras.layers.GlobalAveragePooling2D(dtype="float32")(keras.layers.Add(dtype="float32")([a, b, x]))
        m = keras.Model(x, keras.layers.Dense(4, dtype="float32")(h))
        m.compile(keras.optimizers.SGD(0.01), keras.losses.SparseCategoricalCrossentropy(from_logits=True))
        return m

    gc.collect()
    g = torch.Generator(device="cuda").manual_seed(1)
    batches = [(torch.randn((32, 16, 16, 64), generator=g, device="cuda"), torch.randint(0, 4, (32,), generator=g, device="cuda")) for _ in range(8)]
    losses = []
    for jit in ("auto", False):
        m = build()
        m.jit_compile = jit
        losses.append([float(m.train_on_batch(*b)) for b in batches])
        if jit == "auto":
            assert m._graphed_step.replays > 0 and list(m._graphed_step.input_casts) == [0]
    # the same kernels on the same values; weight gradients are summed by atomics in another order
    assert losses[0] == pytest.approx(losses[1], rel=1e-4)
