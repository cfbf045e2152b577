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


@pytest.mark.parametrize("seqs,new", [(3, 1), (9, 1), (17, 1), (2, 20)])
def test_a_layer_by_either_form_of_its_products(seqs, new, monkeypatch):
    """The head-wise kernels, each beside the library's form of the other, and neither: the same layer but for roundings."""
    from types import SimpleNamespace

    from starter_b200 import ops
    from starter_b200.cache import SequenceCache
    from starter_b200.config import spec as S
    from starter_b200.engine.batch import plan_step
    from starter_b200.parts import lookup

    gen = torch.Generator().manual_seed(seqs)
    spec = S.LatentAttentionSpec(256, 4, 64, 16, 32, 128, 128, 80 ** -0.5, 1e-6, S.InterleavedRopeSpec(16, 1e4), window=None, sink=True,
                                 output_gate=True)
    part = lookup("mixer", spec.kind)(spec, BF, lookup("position", spec.position.kind)(spec.position, BF, "cuda"))
    part.set_params({name: (torch.randn(p.shape, generator=gen) * (p.shape[-1] ** -0.5 if len(p.shape) > 1 else 1.0))
                     .to(torch.float32 if p.role != "matrix" else BF).cuda() for name, p in part.param_specs().items()})
    cache = SequenceCache({0: part.kv_need()}, {0: None}, 128 * seqs, seqs, BF, "cuda")
    slots = [cache.open_sequence() for _ in range(seqs)]
    part.prepare(128)

    def step(tokens):
        arrays = plan_step([SimpleNamespace(slot=s, tokens=[0] * tokens, want=[]) for s in slots], [cache.lengths[s] for s in slots])
        for s in slots:
            cache.reserve(s, cache.lengths[s] + tokens)
            cache.advance(s, tokens)
        cache.sync_table()
        return SimpleNamespace(host=arrays, n_seqs=seqs, max_q_len=tokens, max_kv_len=int(arrays["seq_kv_len"].max()), cache=cache,
                               status=torch.zeros(1, dtype=torch.int32).cuda(), **{k: torch.from_numpy(v).cuda() for k, v in arrays.items()})

    part(torch.randn(seqs * 70, 256, generator=gen).to(BF).cuda(), step(70), 0)
    x, ctx, got = torch.randn(seqs * new, 256, generator=gen).to(BF).cuda(), step(new), {}
    for form in ((False, False), (True, False), (False, True), (True, True)):
        monkeypatch.setattr(ops, "latent_heads_take", lambda *a: form)
        got[form] = part(x, ctx, 0).double()
    want = got[(False, False)]
    for form, y in got.items():
        # a rounding of the queries, of the sums and of the outputs may fall the other way: 2^-8 of single terms each
        assert bool(y.isfinite().all()) and float((y - want).norm()) <= 2.0 ** -7 * float(want.norm())
