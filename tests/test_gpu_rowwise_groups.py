"""The plain attention's two warps a query head, and its four warps up to four heads of a group in steps of many tokens: groups of all
sizes, contexts that end before, at and behind a warp's sixteen keys and a round of sixty-four, windows, head sizes, against float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu
F = torch.float64


@pytest.mark.parametrize("heads,kv_heads,dim,window", [(3, 3, 128, 0), (4, 2, 64, 0), (6, 2, 100, 0), (8, 2, 128, 0), (5, 1, 36, 0), (16, 2, 128, 0),
                                                       (4, 1, 4, 0), (8, 2, 128, 1), (8, 2, 64, 40), (3, 1, 128, 17)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_groups_of_heads(heads, kv_heads, dim, window, dtype):
    against_float64(heads, kv_heads, dim, window, dtype, 1)


# (four heads a block from 1,184 heads of tokens on; groups that leave a block with one to four heads)
@pytest.mark.parametrize("heads,kv_heads,dim,window", [(4, 1, 128, 0), (5, 1, 36, 0), (6, 1, 64, 17), (16, 2, 128, 0), (12, 3, 4, 40), (11, 1, 100, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_four_heads_a_block(heads, kv_heads, dim, window, dtype):
    against_float64(heads, kv_heads, dim, window, dtype, 1 + 1184 // (26 * heads))


def against_float64(heads, kv_heads, dim, window, dtype, copies):
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(heads * dim + window)
    pages, page, table = 12, ops.PAGE_TOKENS, 6
    longest = min(table * page, 200)
    store = [(torch.randn(pages, kv_heads, page, dim, generator=gen) * (2.0 if n else 1.0)).to(dtype).cuda() for n in (0, 1)]
    order = torch.randperm(pages, generator=gen)[:2 * table].view(2, table).to(torch.int32)
    pos = sorted({p for p in (0, 1, 14, 15, 16, 17, 62, 63, 64, 65, 79, 80, 127, 128, longest - 1) if p < longest})
    tok_pos = torch.tensor(pos * 2, dtype=torch.int32)
    tok_slot = torch.tensor([0] * len(pos) + [1] * len(pos), dtype=torch.int32)
    q = torch.randn(len(tok_pos), heads * dim, generator=gen).to(dtype).cuda()
    scale = dim ** -0.5
    if copies > 1:
        assert copies * len(tok_pos) * heads >= 1184
    got = ops.attention_rowwise(q.repeat(copies, 1), *store, order.cuda(), tok_slot.repeat(copies).cuda(), tok_pos.repeat(copies).cuda(), heads,
                                kv_heads, dim, scale, window or None)
    got = got.view(copies, len(tok_pos), -1)
    assert torch.equal(got, got[:1].expand_as(got))
    got = got[0]
    want = torch.empty(len(tok_pos), heads, dim, dtype=F)
    for t, (slot, p) in enumerate(zip(tok_slot.tolist(), tok_pos.tolist())):
        first = max(0, p - window + 1) if window else 0
        k, v = (s.cpu().to(F)[order[slot].long()].transpose(0, 1).reshape(kv_heads, table * page, dim)[:, first:p + 1] for s in store)
        w = torch.softmax(torch.einsum("ghd,gkd->ghk", q[t].cpu().to(F).view(kv_heads, heads // kv_heads, dim) * scale, k), dim=-1)
        want[t] = torch.einsum("ghk,gkd->ghd", w, v).reshape(heads, dim)
    off = (got.cpu().to(F).view_as(want) - want).abs().max()
    # float sums of up to 200 products of unit size, exponentials of 2 ulp; a rounding to bfloat16 is 2^-9 of the result
    assert float(off) <= (2e-6 if dtype == torch.float32 else 2.0 ** -8) * float(want.abs().max())


# keys whose scores are minus infinity: the only key of a warp, all of a warp's first sixteen, all but the last
@pytest.mark.parametrize("heads,kv_heads", [(3, 3), (4, 2), (8, 2)])
@pytest.mark.parametrize("copies", [1, 500])
@pytest.mark.parametrize("pos,gone", [(16, [16]), (32, [32]), (48, [48]), (100, list(range(16, 32)) + list(range(80, 96))), (77, list(range(77)))])
def test_scores_of_minus_infinity_weigh_nothing(heads, kv_heads, pos, gone, copies):
    from starter_b200 import ops

    dim, page = 64, ops.PAGE_TOKENS
    gen = torch.Generator().manual_seed(pos)
    store = [torch.randn(2, kv_heads, page, dim, generator=gen).cuda() for _ in range(2)]
    q = torch.rand(1, heads * dim, generator=gen).cuda() + 0.5
    rows = [store[0][j // page, :, j % page] for j in range(pos + 1)]
    for j in gone:
        rows[j][:, 3] = -float("inf")
    zero = torch.zeros(copies, dtype=torch.int32, device="cuda")
    got = ops.attention_rowwise(q.repeat(copies, 1), *store, torch.tensor([[0, 1]], dtype=torch.int32).cuda(), zero, zero + pos, heads, kv_heads, dim,
                                0.125)
    left = [j for j in range(pos + 1) if j not in gone]
    k, v = (torch.stack([s[j // page, :, j % page] for j in left]).to(F) for s in store)
    s = torch.einsum("hgd,khd->hgk", q.view(kv_heads, heads // kv_heads, dim).to(F) * 0.125, k)
    want = torch.einsum("hgk,khd->hgd", torch.softmax(s, dim=-1), v).reshape(1, -1)
    assert float((got.to(F) - want).abs().max()) <= 2e-6 * float(want.abs().max())
