"""The experts' row kernels where they change form: routing with the logits in registers or read again, choices beyond a warp's lanes, tiles
in equal shares, rows of 16-byte pieces and of single values, few and many rows."""
import pytest
import torch

from iian_b200.ops.cuda_backend import CudaKernels

pytestmark = pytest.mark.gpu
K = CudaKernels


@pytest.mark.parametrize("E,top", [(1, 1), (33, 5), (64, 33), (65, 8), (256, 40), (257, 6), (2048, 3)])
def test_route(E, top):
    g = torch.Generator("cuda").manual_seed(E)
    logits = torch.randn(9, E + 3, device="cuda", generator=g)[:, :E]
    logits[:, E // 2] = logits[:, 0]                                  # a tie goes to the lower number
    ids = torch.full((9, top), -7, device="cuda", dtype=torch.int32)
    w = torch.full((9, top), 7.0, device="cuda")
    K().moe_route(logits, top, ids, w)
    want = torch.sort(logits, dim=1, descending=True, stable=True).indices[:, :top]
    assert torch.equal(ids.long(), want)
    exact = torch.sigmoid(torch.gather(logits, 1, want).double())
    assert ((w.double() - exact).abs() <= 1e-6 * exact).all()         # an exponential, a sum and a quotient in 32 bits


@pytest.mark.parametrize("M,E,rows", [(1, 1, 64), (700, 3, 64), (700, 3, 256), (513, 1, 256), (2000, 70, 128), (40, 200, 256)])
def test_plan(M, E, rows):
    ids = (torch.rand(M, device="cuda", generator=torch.Generator("cuda").manual_seed(M)) ** 2 * E).int()
    most = -(-M // rows) + E
    offsets, pos = torch.full((E + 1,), -7, device="cuda", dtype=torch.int32), torch.full((M,), -7, device="cuda", dtype=torch.int32)
    tiles = torch.full((1 + 2 * most,), -7, device="cuda", dtype=torch.int32)
    K().moe_plan(ids, E, offsets, pos, tiles, rows)
    off, at = offsets.tolist(), pos.tolist()
    assert off == [0] + torch.bincount(ids.long(), minlength=E).cumsum(0).tolist() and sorted(at) == list(range(M))
    assert all(off[e] <= p < off[e + 1] for e, p in zip(ids.tolist(), at))
    t = tiles.tolist()
    assert t[0] <= most
    pairs = [(t[1 + 2 * i], t[2 + 2 * i]) for i in range(t[0])] + [(E, M)]
    seen = 0
    for (e, r), (e2, r2) in zip(pairs, pairs[1:]):                    # the tiles follow one another without a gap, none too long
        assert r == seen and off[e] <= r < off[e + 1]
        seen = r2 if e2 == e else off[e + 1]
        assert 0 < seen - r <= rows
    assert seen == M


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,W,top", [(1, 8, 1), (3, 2048, 5), (127, 1028, 2), (128, 33, 3), (1024, 520, 2), (1025, 4104, 1)])
def test_scatter_and_combine(dtype, n, W, top):
    g = torch.Generator("cuda").manual_seed(n + W)
    h = torch.randn(n, W, device="cuda", generator=g).to(dtype)
    pos = torch.randperm(n * top, device="cuda", generator=g).int()
    w = torch.rand(n * top, device="cuda", generator=g)
    xs = torch.full((n * top, W), 7.0, device="cuda", dtype=dtype)
    K().moe_scatter(h, pos, w, xs, top)
    assert torch.equal(xs[pos.long()], (h.float().repeat_interleave(top, 0) * w[:, None]).to(dtype))
    out = torch.full((n, W), 7.0, device="cuda", dtype=dtype)
    K().moe_combine(xs, pos, out, top, w)
    terms = xs[pos.long()].double().view(n, top, W) * w.double().view(n, top, 1)
    eps = top * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)          # 32-bit sums of `top` terms, rounded once
    assert ((out.double() - terms.sum(1)).abs() <= eps * 1.01 * terms.abs().sum(1) + 1e-30).all()
