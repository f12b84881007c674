"""The variants a dispatch rule chooses between, each at the sizes where it can go wrong (needs a B200)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,V,ld", [(1, 64, 64), (77, 64, 64), (513, 65, 72), (100, 100, 100), (33, 129, 136), (7, 1000, 1000), (19, 2047, 2047),
                                       (9, 2048, 2048), (5, 2049, 2056)])
def test_cross_entropy_of_narrow_and_wide_rows(rows, V, ld, dtype):
    from keras_b200.kernels import ops as kops

    torch.manual_seed(V)
    buf = (torch.randn(rows, ld, device="cuda") * 3).to(dtype)
    if V > 70:
        buf[:, 3:17] = float("-inf")  # masked classes
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
@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (264, 520, 1000), (136, 1000, 72), (2664, 512, 520), (2049 * 8, 264, 136)])
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
                                           K_._i(fp32), K_._i(split), K_._i(variant), K_._p(err), K_._stream())
            K_._check(code, "gemm_bf16")
            want = torch.relu(ref + bias) if with_bias else ref + 2.0 if add else ref
            rel = ((c.double() - want).norm() / want.norm()).item()
            # fp32 sums of K exact products (2^-24 each), one rounding to bf16 (2^-9)
            assert rel < (2.0 ** -17 if fp32 else 2.0 ** -8), (a_mn, b_mn, split, fp32, rel)
            assert int(err.item()) == 0
