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
