"""The head-wise products around the attention over cached latents: against float64, at the edges of their blocks of tokens, columns
and k-steps, from one part and from many (some without a key), with and without a sink and a gate."""

import pytest
import torch

pytestmark = pytest.mark.gpu
BF, F = torch.bfloat16, torch.float64


@pytest.mark.parametrize("n", [1, 15, 16, 17, 64])
@pytest.mark.parametrize("heads,dim,rot,rank,layout", [(16, 128, 64, 512, "interleaved"), (3, 16, 8, 64, "half_split"),
                                                       (2, 240, 16, 192, "interleaved")])
def test_fold(n, heads, dim, rot, rank, layout):
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(n + dim)
    q = torch.randn(n, heads * (dim + rot), generator=gen).to(BF).cuda()
    uk = (torch.randn(heads * dim, rank, generator=gen) * dim ** -0.5).to(BF).cuda()
    angle = torch.randn(100, rot // 2, generator=gen)
    cos, sin, pos = angle.cos().cuda(), angle.sin().cuda(), torch.randint(0, 100, (n,), generator=gen).to(torch.int32).cuda()
    got = ops.latent_fold(q, uk, cos, sin, pos, heads, dim, rot, rot, rank, layout)
    q3 = q.view(n, heads, dim + rot)
    want = torch.einsum("thd,hdr->thr", q3[..., :dim].to(F), uk.view(heads, dim, rank).to(F))
    # float sums of up to 240 products, one rounding to bfloat16
    assert float((got[..., :rank].double() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max())
    turned = torch.zeros_like(got)
    ops.latent_rotate_q(q, turned, cos, sin, pos, heads, dim, rot, rot, rank, layout)
    assert torch.equal(got[..., rank:], turned[..., rank:])


@pytest.mark.parametrize("n", [1, 16, 17, 40])
@pytest.mark.parametrize("parts", [1, 2, 9, 32])
@pytest.mark.parametrize("heads,rank,vdim,sink,gate", [(16, 512, 128, True, True), (2, 64, 8, False, False), (3, 192, 40, True, False),
                                                       (3, 448, 72, False, True)])
def test_unfold(n, parts, heads, rank, vdim, sink, gate):
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(n + parts + rank)
    uv = (torch.randn(heads * vdim, rank, generator=gen) * rank ** -0.5).to(BF).cuda()
    wide = torch.randn(n, heads * vdim + 8, generator=gen).to(BF).cuda() if gate else None
    sk = torch.linspace(-1.0, 1.0, heads).cuda() if sink else None
    if parts == 1:
        summed = torch.randn(n, heads, rank, generator=gen).to(BF).cuda()
        given, rows = (summed, None, None), summed.to(F)
    else:
        ref = torch.randn(parts, n * heads, generator=gen) * 3.0
        weight = torch.rand(parts, n * heads, generator=gen) + 0.5
        acc = torch.randn(parts, n * heads, rank, generator=gen)
        ref[-1, 0], weight[-1, 0], acc[-1, 0] = float("-inf"), 0.0, 0.0              # a part in which a row sees no key
        given = (None, acc.cuda(), torch.stack([ref, weight], dim=2).contiguous().cuda())
        own = (sk.cpu() if sink else torch.full((heads,), float("-inf"))).repeat(n).to(F)
        top = torch.maximum(ref.to(F).max(dim=0).values, own)
        e = torch.exp(ref.to(F) - top)
        total = (e * weight.to(F)).sum(0) + (torch.exp(own - top) if sink else 0.0)
        rows = ((e / total)[:, :, None] * acc.to(F)).sum(0).view(n, heads, rank).to(BF).to(F).cuda()
    got = ops.latent_unfold(given, uv, heads, vdim, rank, sk, wide, 8 if gate else 0).double()
    want = torch.einsum("thr,hvr->thv", rows, uv.view(heads, vdim, rank).to(F)).reshape(n, heads * vdim)
    if gate:
        want = want * torch.sigmoid(wide[:, 8:].to(F))
    # the joined rows may round the other way (2^-8 of single terms), then two roundings of the result
    assert float((got - want).abs().max()) <= 2.0 ** -7 * float(want.abs().max())
    assert float((got - want).norm()) <= 2.0 ** -8 * float(want.norm())
