"""The sampling kernel at the sizes where its cluster of CTAs, its slices and its searches change form: one CTA, two, eight with a
ragged last slice, slices too large for shared memory; ties, entries of minus infinity and NaN, single candidates."""
import pytest
import torch

import plain_qwen3 as plain
from iian_b200 import ops

pytestmark = pytest.mark.gpu

SETTINGS = [(0.7, 20, 0.8, 0.0), (1.0, 0, 1.0, 0.0), (0.8, 0, 0.9, 0.0), (1.0, 0, 1.0, 0.05), (1.3, 1, 1.0, 0.0), (0.0, 0, 1.0, 0.0),
            (1.0, 50, 0.3, 0.01), (1.0, 0, 0.0, 0.0), (0.5, 0, 1e-6, 0.0), (1.0, 0, 0.999999, 0.0)]


def draw(logits, settings, u):
    f = lambda i, dt: torch.tensor([s[i] for s in settings], dtype=dt).cuda()
    out = torch.full((len(settings),), -7, dtype=torch.int32).cuda()
    ops.kernels().sample(logits.cuda(), f(0, torch.float32), f(1, torch.int32), f(2, torch.float32), f(3, torch.float32), u.cuda(), out)
    return out.tolist()


@pytest.mark.parametrize("V", [1, 7, 4096, 4097, 8193, 32768 + 5, 151936, 8 * 50 * 1024 + 9])
def test_draws_land_in_their_interval(V):
    g = torch.Generator().manual_seed(V)
    logits = torch.randn(len(SETTINGS), V, generator=g) * 2.5
    if V > 100:
        logits[:, 3::11] = float("-inf")
        logits[1:, [10, V // 2, V - 2]] = logits.max() + 0.25           # ties at the top, in different slices
        logits[2, 40:60] = logits[2, 40]                                  # and further down
    u = torch.rand(len(SETTINGS), generator=g)
    u[0], u[1] = 0.0, 1.0 - 2.0 ** -24
    got = draw(logits, SETTINGS, u)
    for r, (T, top_k, top_p, min_p) in enumerate(SETTINGS):
        if T < 1e-5 or top_p <= 0.0:
            assert got[r] == plain.argmax(logits[r])
            continue
        probs = plain.candidate_probs(logits[r], T, top_k, top_p, min_p)
        # the kernel takes the running mass in 64 bits; the oracle's 32-bit sums of V terms differ from it by V * 2^-24 of the total at
        # most, in practice far less: 1e-5 as in the other sampling test
        cum = torch.cumsum(probs.double(), 0)
        total, target = cum[-1].item(), u[r].item() * cum[-1].item()
        hi = cum[got[r]].item()
        assert probs[got[r]] > 0 and hi - probs[got[r]].item() - 1e-5 * total <= target <= hi + 1e-5 * total, f"row {r}"
    alone = [draw(logits[r: r + 1], SETTINGS[r: r + 1], u[r: r + 1])[0] for r in range(len(SETTINGS))]
    assert alone == got                                                     # whatever else is in the batch


def test_rows_without_a_largest_value():
    inf = float("inf")
    logits = torch.zeros(4, 5000)
    logits[0] = -inf
    logits[1] = float("nan")
    logits[2, 4999] = inf
    logits[3] = float("nan")
    logits[3, 4500] = -3.0
    s = [(1.0, 5, 0.9, 0.0)] * 4
    assert draw(logits, s, torch.full((4,), 0.5)) == [0, 0, 4999, 4500]


@pytest.mark.parametrize("V,low,high", [(3000, 5, 2000), (3000, 2000, 5), (40000, 5, 39990)])
def test_the_two_zeros_are_one_value(V, low, high):
    """A largest value held by a -0.0 (at ``low``) and a +0.0 (at ``high``): ties, the lower id first."""
    logits = torch.full((6, V), -60.0)
    logits[:, low], logits[:, high] = -0.0, 0.0
    a, b = sorted((low, high))
    s = [(1.0, 1, 1.0, 0.0), (1.0, 2, 1.0, 0.0), (1.0, 0, 0.3, 0.0), (1.0, 0, 0.9, 0.0), (1.0, 0, 0.9, 0.0), (0.0, 0, 1.0, 0.0)]
    assert draw(logits, s, torch.tensor([0.9, 0.9, 0.9, 0.9, 0.1, 0.5])) == [a, b, a, b, a, a]
