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
                                   (40, 6, 176), (64, 4, 48), (5, 6, 68), (9, 3, 260)])
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
