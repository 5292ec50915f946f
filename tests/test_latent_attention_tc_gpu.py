"""Attention over a cached latent for portions of prompts on tcgen05 against float64: row tiles that end inside a request, key tiles that
end inside a page, windows, both ranks, widths with and without chunks outside the values; what lies in the cache behind the newest key (here
NaN) must not reach the output."""
from types import SimpleNamespace

import pytest
import torch

from iian_b200.ops.cuda_backend import CudaKernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank,rot,heads,page", [(512, 64, 16, 16), (512, 64, 5, 64), (512, 0, 16, 8), (256, 64, 3, 32), (256, 0, 128, 16)])
@pytest.mark.parametrize("cached,news,window", [([0], [64], 0), ([0, 70, 5], [130, 33, 1], 0), ([200, 63, 0], [65, 64, 63], 50),
                                                ([17] * 40, [1 + i % 9 for i in range(40)], 0), ([100 + 61 * i for i in range(50)], [1] * 50, 0)])
def test_portions_against_float64(rank, rot, heads, page, cached, news, window):
    g = torch.Generator("cuda").manual_seed(rank + heads + len(news))
    width, n = rank + rot, sum(news)
    blocks = [-(-(c + m) // page) for c, m in zip(cached, news)]
    order = torch.randperm(sum(blocks) + 1, generator=torch.Generator().manual_seed(7)).tolist()
    rows = torch.full((sum(blocks) + 1, page, width), float("nan"), device="cuda", dtype=torch.bfloat16)
    bt = torch.full((len(news), max(blocks)), -1, dtype=torch.int32)
    q = (2 * torch.randn(n, heads, width, device="cuda", generator=g)).bfloat16()
    sink = torch.randn(heads, device="cuda", generator=g)
    scale, cu, want, bound = width ** -0.5, [0], [], []
    for i, (c, m) in enumerate(zip(cached, news)):
        keys = torch.randn(c + m, width, device="cuda", generator=g).bfloat16()
        for b in range(blocks[i]):
            bt[i, b] = order.pop()
            part = keys[b * page: (b + 1) * page]
            rows[int(bt[i, b]), : len(part)] = part
        pos, j = torch.arange(c, c + m, device="cuda")[:, None], torch.arange(c + m, device="cuda")[None]
        hidden = (j > pos) | (pos - j >= window if window else False)
        z = torch.einsum("thw,kw->thk", q[cu[-1]: cu[-1] + m].double(), keys.double()) * scale
        z = torch.cat([z.masked_fill(hidden[:, None], float("-inf")), sink.double()[None, :, None].expand(m, -1, 1)], 2)
        p = torch.softmax(z, 2)[..., :-1]
        want.append(p @ keys[:, :rank].double())
        bound.append(p @ keys[:, :rank].double().abs())
        cu.append(cu[-1] + m)
    cuda = lambda x: torch.as_tensor(x, dtype=torch.int32).cuda()
    meta = SimpleNamespace(cu_q=cuda(cu), ctx_len=cuda([c + m for c, m in zip(cached, news)]), block_table=bt.cuda(), num_seqs=len(news),
                           max_q_len=max(news), seq_of_token=cuda([i for i, m in enumerate(news) for _ in range(m)]))
    K, outs = CudaKernels(), []
    for parts in (1, 2, 5):                    # the keys whole and cut; parts without keys among them
        outs.append(torch.full((n, heads, rank), 7.0, device="cuda", dtype=torch.bfloat16))
        K.latent_attention_tc(q, rows, outs[-1], sink, meta, num_heads=heads, rank=rank, scale=scale, window=window or None, parts=parts)
        K.tcgen05_check(q.device)
    # the weights and the result are rounded to bfloat16, whose significand has 8 bits: by 2^-8 of each term and 2^-8 of the sum at most;
    # the scores are 32-bit sums of up to 576 products whose exponentials are off by 1e-4 at most
    want, bound = torch.cat(want), torch.cat(bound)
    for out in outs:
        assert bool(((out.double() - want).abs() <= (2.0 ** -7 + 2e-4) * bound).all())


@pytest.mark.parametrize("rank,rot,heads", [(512, 64, 16), (256, 0, 16), (256, 64, 3)])
@pytest.mark.parametrize("parts", [1, 3])
def test_tokens_without_a_key_give_zeros(rank, rot, heads, parts):
    """Long portions of requests that have no context, or less than they have tokens: rows before the first key are zeros, as the other kernel
    writes them; the rest sees what there is."""
    g = torch.Generator("cuda").manual_seed(rank + heads)
    width, page, news, ctx = rank + rot, 16, [100, 90, 130, 1], [0, 33, 0, 0]
    n = sum(news)
    rows = torch.randn(3, page, width, device="cuda", generator=g).bfloat16()
    q = torch.randn(n, heads, width, device="cuda", generator=g).bfloat16()
    sink = torch.randn(heads, device="cuda", generator=g)
    cuda = lambda x: torch.as_tensor(x, dtype=torch.int32).cuda()
    meta = SimpleNamespace(cu_q=cuda([0, 100, 190, 320, 321]), ctx_len=cuda(ctx), block_table=cuda([[-1] * 3, [0, 1, 2], [-1] * 3, [-1] * 3]), num_seqs=4,
                           max_q_len=130, max_ctx=130, seq_of_token=cuda([i for i, m in enumerate(news) for _ in range(m)]))
    K, out = CudaKernels(), torch.full((n, heads, rank), 7.0, device="cuda", dtype=torch.bfloat16)
    K.latent_attention_tc(q, rows, out, sink, meta, num_heads=heads, rank=rank, scale=width ** -0.5, window=None, parts=parts)
    K.tcgen05_check(q.device)
    assert not out[:157].any() and not out[190:].any()              # the second request's first 57 tokens lie before its first key
    keys = rows.view(-1, width)[:33].double()
    z = torch.einsum("thw,kw->thk", q[157:190].double(), keys) * width ** -0.5
    z = z.masked_fill(torch.arange(33, device="cuda")[None, None] > torch.arange(33, device="cuda")[:, None, None], float("-inf"))
    p = torch.softmax(torch.cat([z, sink.double()[None, :, None].expand(33, -1, 1)], 2), 2)[..., :-1]
    # as above
    assert bool(((out[157:190].double() - p @ keys[:, :rank]).abs() <= (2.0 ** -7 + 2e-4) * (p @ keys[:, :rank].abs())).all())


@pytest.mark.parametrize("rank,heads,page", [(512, 16, 16), (512, 8, 64), (512, 13, 8), (256, 16, 128), (256, 5, 16), (256, 16, 32)])
@pytest.mark.parametrize("contexts,window", [([64, 1, 128, 129], 0), ([300] * 40, 0), ([40 + 97 * i for i in range(33)], 0), ([5000, 17, 3, 900], 0),
                                             ([700, 130, 20, 128, 4000], 128), ([1 + 61 * i for i in range(170)], 1000)])
def test_decoded_tokens_with_keys_as_rows(rank, heads, page, contexts, window):
    """The line of key tiles over the CTAs: sequences of one tile and of many, cut by a CTA's border or not, padding and a request without
    context among them, the last page NaN behind the newest key."""
    g = torch.Generator("cuda").manual_seed(rank + heads + len(contexts))
    width, n = rank + 64, len(contexts) + 2                        # a request without context and a padding token at the end
    blocks = [-(-c // page) for c in contexts]
    order = torch.randperm(sum(blocks) + 1, generator=torch.Generator().manual_seed(7)).tolist()
    rows = torch.full((sum(blocks) + 1, page, width), float("nan"), device="cuda", dtype=torch.bfloat16)
    bt = torch.full((n, max(blocks)), -1, dtype=torch.int32)
    q = (2 * torch.randn(n, heads, width, device="cuda", generator=g)).bfloat16()
    sink = torch.randn(heads, device="cuda", generator=g)
    scale, want, bound = width ** -0.5, [], []
    for i, c in enumerate(contexts):
        keys = torch.randn(c, width, device="cuda", generator=g).bfloat16()
        for b in range(blocks[i]):
            bt[i, b] = order.pop()
            part = keys[b * page: (b + 1) * page]
            rows[int(bt[i, b]), : len(part)] = part
        z = (q[i].double() @ keys.double().T) * scale
        if window:
            z[:, : max(0, c - window)] = float("-inf")
        p = torch.softmax(torch.cat([z, sink.double()[:, None]], 1), 1)[:, :-1]
        want.append(p @ keys[:, :rank].double())
        bound.append(p @ keys[:, :rank].double().abs())
    cuda = lambda x: torch.as_tensor(x, dtype=torch.int32).cuda()
    meta = SimpleNamespace(cu_q=cuda(list(range(n + 1))), ctx_len=cuda(contexts + [0, 1]), block_table=bt.cuda(), num_seqs=n, max_q_len=1,
                           seq_of_token=cuda(list(range(n - 1)) + [-1]))
    K, out = CudaKernels(), torch.full((n, heads, rank), 7.0, device="cuda", dtype=torch.bfloat16)
    assert K.latent_line_ok(q, rows, rank, scale)
    K.latent_line(q, rows, out, sink, meta, num_heads=heads, rank=rank, scale=scale, window=window or None)
    K.tcgen05_check(q.device)
    assert not out[-2:].any()
    # as above
    assert bool(((out[:-2].double() - torch.stack(want)).abs() <= (2.0 ** -7 + 2e-4) * torch.stack(bound)).all())


@pytest.mark.parametrize("rank,heads,contexts", [(512, 16, [800, 2400, 1600]), (256, 16, [3000, 900]), (512, 3, [130, 64, 2000, 5000, 257, 31])])
def test_decoded_tokens_weights_keep_more_than_16_bits(rank, heads, contexts):
    """The error against 64 bits is the result's own rounding to bfloat16 and little more: weights in two parts are good to 2^-17, sums of
    products to 2^-20 or so, against 2^-9.  One bfloat16 part each would add 2^-9 / sqrt(3) of the root mean square, some 15 percent here."""
    g = torch.Generator("cuda").manual_seed(rank + heads)
    width, n, page = rank + 64, len(contexts), 16
    rows = torch.randn(sum(-(-c // page) for c in contexts), page, width, device="cuda", generator=g).bfloat16()
    bt, at, want = torch.full((n, -(-max(contexts) // page)), -1, dtype=torch.int32), 0, []
    q = torch.randn(n, heads, width, device="cuda", generator=g).bfloat16()
    for i, c in enumerate(contexts):
        pages = -(-c // page)
        bt[i, :pages] = torch.arange(at, at + pages)
        keys = rows[at: at + pages].view(-1, width)[:c].double()
        at += pages
        want.append(torch.softmax(q[i].double() @ keys.T * width ** -0.5, 1) @ keys[:, :rank])
    want = torch.stack(want)
    cuda = lambda x: torch.as_tensor(x, dtype=torch.int32).cuda()
    meta = SimpleNamespace(cu_q=cuda(list(range(n + 1))), ctx_len=cuda(contexts), block_table=bt.cuda(), num_seqs=n, max_q_len=1,
                           seq_of_token=cuda(list(range(n))))
    K, out = CudaKernels(), torch.empty(n, heads, rank, device="cuda", dtype=torch.bfloat16)
    K.latent_line(q, rows, out, None, meta, num_heads=heads, rank=rank, scale=width ** -0.5, window=None)
    K.tcgen05_check(q.device)
    assert (out.double() - want).norm() < 1.02 * (want.bfloat16().double() - want).norm()
