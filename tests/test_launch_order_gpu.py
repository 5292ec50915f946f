"""Attention whose CTAs take their work in falling order of length, against float64: decode batches just above and below the sizes that are
ranked, with equal contexts among them; portions of one to ninety requests, empty row tiles and equal lengths among them."""
from types import SimpleNamespace

import pytest
import torch

from iian_b200.ops.cuda_backend import CudaKernels

pytestmark = pytest.mark.gpu


def case(ctx, news, nh, nkv, page=16, hd=128):
    g = torch.Generator("cuda").manual_seed(len(ctx) + nkv)
    blocks = [-(-c // page) for c in ctx]
    order = torch.randperm(sum(blocks), generator=torch.Generator().manual_seed(3)).tolist()
    k = torch.randn(sum(blocks), nkv, page, hd, device="cuda", generator=g).bfloat16()
    v = torch.randn(sum(blocks), nkv, page, hd, device="cuda", generator=g).bfloat16()
    q = torch.randn(sum(news), nh, hd, device="cuda", generator=g).bfloat16()
    bt = torch.full((len(ctx), max(blocks)), -1, dtype=torch.int32)
    cu, pos, seq, want, bound = [0], [], [], [], []
    for i, (c, n) in enumerate(zip(ctx, news)):
        mine = [order.pop() for _ in range(blocks[i])]
        bt[i, : blocks[i]] = torch.tensor(mine)
        flat = lambda x: x[mine].transpose(0, 1).reshape(nkv, -1, hd)[:, :c].double().repeat_interleave(nh // nkv, 0)
        z = torch.einsum("thd,hkd->htk", q[cu[-1]: cu[-1] + n].double(), flat(k)) * hd ** -0.5
        p = torch.softmax(z.masked_fill(torch.arange(c, device="cuda")[None, None] > torch.arange(c - n, c, device="cuda")[None, :, None],
                                        float("-inf")), 2)
        want.append((p @ flat(v)).transpose(0, 1).reshape(n, -1))
        bound.append((p @ flat(v).abs()).transpose(0, 1).reshape(n, -1))
        cu.append(cu[-1] + n)
        pos += range(c - n, c)
        seq += [i] * n
    cuda = lambda x: torch.tensor(x, dtype=torch.int32).cuda()
    meta = SimpleNamespace(cu_q=cuda(cu), ctx_len=cuda(ctx), block_table=bt.cuda(), positions=cuda(pos), seq_of_token=cuda(seq),
                           num_seqs=len(ctx), max_q_len=max(news), max_ctx=max(ctx), decode_only=max(news) == 1)
    return q, k, v, meta, torch.cat(want), torch.cat(bound)


def check(out, want, bound):
    # the weights and the result are rounded to bfloat16 (2^-8 of each term and of the sum at most); the scores are 32-bit sums of 128
    # products whose exponentials are off by 1e-4 at most
    assert bool(((out.double() - want).abs() <= (2.0 ** -7 + 2e-4) * bound).all())


@pytest.mark.parametrize("contexts", [lambda i: 1 + (i * 131) % 700 if i % 5 else 333, lambda i: 40, lambda i: 3000 if i == 7 else 1 + i % 3,
                                      lambda i: 1 << (i % 11)])
@pytest.mark.parametrize("S,nkv", [(37, 8), (38, 8), (56, 8), (64, 8), (256, 2), (257, 2), (130, 4)])
def test_decode_in_falling_order_of_contexts(S, nkv, contexts):
    ctx = [contexts(i) for i in range(S)]
    q, k, v, meta, want, bound = case(ctx, [1] * S, 2 * nkv, nkv)
    out = torch.full((S, 2 * nkv * 128), 7.0, device="cuda", dtype=torch.bfloat16)
    CudaKernels().paged_attention_mma(q, k, v, out, meta, num_heads=2 * nkv, num_kv_heads=nkv, head_dim=128, scale=128 ** -0.5, window=None,
                                      n_split=1)
    check(out, want, bound)


@pytest.mark.parametrize("cached,news", [([0], [300]), ([500, 0, 3], [33, 260, 1]), ([64] * 33, [64] * 33),
                                         ([(i * 37) % 300 for i in range(90)], [1 + (i * 53) % 70 for i in range(90)]),
                                         ([2000, 0] + [(i * 97) % 900 for i in range(150)], [65, 200] + [1 + (i * 53) % 70 for i in range(150)]),
                                         ([7] * 40, [65 + i % 2 for i in range(40)]), ([(i * 211) % 1500 for i in range(140)], [1] * 139 + [129])])
def test_portions_in_falling_order_of_their_keys(cached, news):
    q, k, v, meta, want, bound = case([c + n for c, n in zip(cached, news)], news, 8, 2)
    K, out = CudaKernels(), torch.full((sum(news), 8 * 128), 7.0, device="cuda", dtype=torch.bfloat16)
    K.paged_attention_tc(q, k, v, out, meta, num_heads=8, num_kv_heads=2, head_dim=128, scale=128 ** -0.5, window=None)
    K.tcgen05_check(q.device)
    check(out, want, bound)
