"""The delta rule over portions of prompts in bfloat16 models.  The scan four tokens at a time against the scan token by token: lengths around
multiples of four and of a stage, sequences of a single token and padding between long ones, states that go on, the step whole and in
segments.  The preparation of steps of many tokens against steps of few, bit for bit."""
from types import SimpleNamespace

import pytest
import torch

from iian_b200.ops.cuda_backend import CudaKernels

pytestmark = pytest.mark.gpu


def walk(blocks, scratch, lens, H, G, D, V, per_head, told=False):
    """(outputs of two steps, states, what ``_delta_pieces`` chose); ``told``: the lengths are known on the host too."""
    K, chosen = CudaKernels(), []
    K._delta_pieces = lambda *a: chosen.append(CudaKernels._delta_pieces(K, *a)) or chosen[-1]
    g = torch.Generator("cuda").manual_seed(sum(lens) + D + H)
    C = 2 * G * D + H * V
    state = torch.randn(len(lens) + 1, K.delta_state_floats(H, G, D, V, 4), device="cuda", generator=g)
    taps = torch.randn(C, 4, device="cuda", generator=g) * 0.4
    a_log, z_width = torch.rand(H, device="cuda", generator=g) * 2.5, H if per_head else H * D
    dt_bias = torch.randn(z_width, device="cuda", generator=g) - 2.0
    slots = [i if i != 1 else -1 for i in range(len(lens))]                       # the second sequence is padding
    bufs, outs = {}, []
    for _ in range(2):                                                              # the second step goes on from the first one's states
        n = sum(lens)
        proj = torch.randn(n, C + H, device="cuda", generator=g).bfloat16()
        z = torch.randn(n, z_width, device="cuda", generator=g)
        cu = [0]
        for x in lens:
            cu.append(cu[-1] + x)
        seq = torch.tensor([i if slots[i] >= 0 else -1 for i, x in enumerate(lens) for _ in range(x)], dtype=torch.int32, device="cuda")
        ctx = SimpleNamespace(cu_q=torch.tensor(cu, dtype=torch.int32, device="cuda"), seq_of_token=seq, max_q_len=max(lens),
                              state_slots=torch.tensor(slots, dtype=torch.int32, device="cuda"), h_q_len=list(lens) if told else [],
                              buf=lambda name, shape, dt: bufs.setdefault((name, tuple(shape)), torch.zeros(shape, dtype=dt, device="cuda")))
        out = torch.full((n, H * V), 7.0, device="cuda")
        K.DELTA_BLOCKS, K.DELTA_BLOCK_BYTES, K.DELTA_SEGMENT_MIN_PIECES = blocks, scratch, 8
        K.delta_rule(proj, 0, C, z, taps, a_log, dt_bias, state, ctx, out, num_heads=H, num_kv_heads=G, dim=D, v_dim=V)
        outs.append(out)
    return outs, state, set(chosen)


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("H,G,D,V", [(4, 2, 128, 128), (3, 3, 64, 48), (2, 1, 128, 16)])
@pytest.mark.parametrize("lens", [[32], [33, 3, 1], [1, 2, 47, 1, 64], [35, 1, 130], [132], [133, 3, 1], [1, 2, 147, 1, 64], [40, 33, 70]])
def test_four_tokens_at_a_time(lens, H, G, D, V, per_head):
    want, want_state, none = walk(False, 0, lens, H, G, D, V, per_head)
    assert none == {None}
    piece = 4 * H * (13 * D + 28)
    cut = sum(lens) // 4 + len(lens) > 8 * len(lens)              # more pieces than eight per sequence
    for scratch, pieces, told in ((192 << 20, 0, False), (192 << 20, 0, True), (piece * 8 * len(lens), 8 if cut else 0, False)):
        got, state, chosen = walk(True, scratch, lens, H, G, D, V, per_head, told)
        assert chosen == {pieces}                                 # the whole step at once, and in segments of eight pieces
        # both are 32-bit sums of the same terms in another order: D of them in a dot product, the sequence's tokens in the state
        for a, b in ((torch.cat(got), torch.cat(want)), (state, want_state)):
            assert (a - b).norm() <= 1e-5 * b.norm() and (a - b).abs().max() <= 1e-4 * b.abs().max()
        at = 0
        for i, n in enumerate(lens):                              # short portions are walked token by token beside long ones too
            if n < CudaKernels.DELTA_BLOCK_MIN_TOKENS:
                assert all(torch.equal(a[at: at + n], b[at: at + n]) for a, b in zip(got, want)) and torch.equal(state[i], want_state[i])
            at += n


def test_short_segments_are_walked_token_by_token():
    K, state = CudaKernels(), torch.zeros(1, 4, device="cuda")
    K.DELTA_BLOCK_BYTES = 4 * K._delta_block_floats(32, 128) * 900
    choose = lambda n, s: K._delta_pieces(1, n, s, 32, 128, 128, 2048, state)
    assert [choose(3000, 10), choose(3800, 1), choose(4096, 4), choose(3648, 101)] == [0, 512, 128, None]


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("given", [False, True])
@pytest.mark.parametrize("H,G,V", [(4, 2, 128), (2, 2, 256), (3, 1, 128)])
def test_preparation_of_many_tokens_gives_the_bits_of_few(H, G, V, given, per_head):
    """Sequences that begin inside a tile of 16 rows, states and convolution tails that are not zero, padding in between, write strengths out
    of the projections or given: one step of 475 tokens against steps of 100 at most, one sequence each."""
    K, D, off = CudaKernels(), 128, 8
    K.DELTA_BLOCKS = False
    g = torch.Generator("cuda").manual_seed(H + V)
    lens, slots, C = [5, 300, 3, 37, 130], [3, 0, -1, 1, 2], 2 * G * D + H * V
    n, zw = sum(lens), H if per_head else H * D
    state0 = torch.randn(4, K.delta_state_floats(H, G, D, V, 4), device="cuda", generator=g)
    proj = torch.randn(n, off + C + H + (-(C + H)) % 8, device="cuda", generator=g).bfloat16()
    both = torch.randn(n, zw + H + (-(zw + H)) % 4, device="cuda", generator=g)
    taps = torch.randn(C, 4, device="cuda", generator=g) * 0.4
    a_log, dt_bias = torch.rand(H, device="cuda", generator=g) * 2.5, torch.randn(zw, device="cuda", generator=g) - 2.0

    def step(rows, cu, seq, which, state, out):
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
        bufs = {}
        ctx = SimpleNamespace(cu_q=i32(cu), seq_of_token=i32(seq), state_slots=i32(which), max_q_len=max(b - a for a, b in zip(cu, cu[1:])),
                              buf=lambda name, shape, dt: bufs.setdefault(name, torch.full(shape, float("nan"), dtype=dt, device="cuda")))
        K.delta_rule(proj[rows], off, off + C, both[rows, :zw], taps, a_log, dt_bias, state, ctx, out[rows], num_heads=H, num_kv_heads=G, dim=D,
                     v_dim=V, b_pre=both[rows, zw: zw + H] if given else None)

    cu = [0]
    for m in lens:
        cu.append(cu[-1] + m)
    whole, few = state0.clone(), state0.clone()
    a, b = torch.full((n, H * V), 7.0, device="cuda"), torch.zeros(n, H * V, device="cuda")
    step(slice(0, n), cu, [i if slots[i] >= 0 else -1 for i, m in enumerate(lens) for _ in range(m)], slots, whole, a)
    for i, m in enumerate(lens):
        for lo in range(0, m if slots[i] >= 0 else 0, 100):
            k = min(100, m - lo)
            step(slice(cu[i] + lo, cu[i] + lo + k), [0, k], [0] * k, [slots[i]], few, b)
    assert torch.equal(whole, few) and torch.equal(a, b)


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("H,G,D,V,lens", [(4, 2, 128, 128, [60, 47, 33, 61, 44]), (4, 2, 128, 128, [33 + i % 9 for i in range(12)]),
                                          (3, 3, 64, 48, [70] + [32 + i for i in range(16)]), (3, 1, 64, 48, [35 + i for i in range(17)])])
def test_forms_of_the_walk_give_the_same_bits(H, G, D, V, lens, per_head):
    """Sequences side by side, more CTAs than SMs, two pieces a stage (the first and third) or one, against each sequence alone, where a warp of
    its own copies the pieces and their vectors are read a step ahead."""
    K, chosen = CudaKernels(), []
    K._delta_pieces = lambda *a: chosen.append(CudaKernels._delta_pieces(K, *a)) or chosen[-1]
    g = torch.Generator("cuda").manual_seed(H + D + len(lens))
    C, n, S, zw = 2 * G * D + H * V, sum(lens), len(lens), H if per_head else H * D
    assert V // 16 * H * S > 148 >= V // 16 * H
    state0 = torch.randn(S, K.delta_state_floats(H, G, D, V, 4), device="cuda", generator=g)
    proj, z = torch.randn(n, C + H, device="cuda", generator=g).bfloat16(), torch.randn(n, zw, device="cuda", generator=g)
    taps = torch.randn(C, 4, device="cuda", generator=g) * 0.4
    a_log, dt_bias = torch.rand(H, device="cuda", generator=g) * 2.5, torch.randn(zw, device="cuda", generator=g) - 2.0

    def step(rows, which, state, out):
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
        mine, cu, bufs = [lens[i] for i in which], [0], {}
        for m in mine:
            cu.append(cu[-1] + m)
        ctx = SimpleNamespace(cu_q=i32(cu), seq_of_token=i32([i for i, m in enumerate(mine) for _ in range(m)]), state_slots=i32(which), max_q_len=max(mine),
                              buf=lambda name, shape, dt: bufs.setdefault(name, torch.full(shape, float("nan"), dtype=dt, device="cuda")))
        K.delta_rule(proj[rows], 0, C, z[rows], taps, a_log, dt_bias, state, ctx, out[rows], num_heads=H, num_kv_heads=G, dim=D, v_dim=V)

    whole, alone = state0.clone(), state0.clone()
    a, b = (torch.full((n, H * V), float("nan"), device="cuda") for _ in range(2))
    step(slice(0, n), list(range(S)), whole, a)
    at = 0
    for i, m in enumerate(lens):
        step(slice(at, at + m), [i], alone, b)
        at += m
    assert set(chosen) == {0} and torch.equal(a, b) and torch.equal(whole, alone)
