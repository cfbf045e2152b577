"""Row kernels of prompts where their pieces, chunks and alignments change: norms that keep a row in registers, packed rotary products,
convolutions of 16 tokens a thread, rotated queries in pieces."""

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
HALF_STEP = 2.0 ** -8 * 1.01     # rounding to bfloat16 and a little for the sums in 32 bits


def ints(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


# a lane's pieces of 8 (bfloat16) or 4 (float): at and beyond 8, 12 and 16 of them
@pytest.mark.parametrize("dtype, hidden", [(BF, 2048), (BF, 2056), (BF, 3072), (BF, 3080), (BF, 4096), (BF, 4104),
                                           (torch.float32, 1024), (torch.float32, 1540), (torch.float32, 2048), (torch.float32, 2052)])
@pytest.mark.parametrize("add", [False, True])
def test_norms_of_many_rows(dtype, hidden, add):
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(hidden)
    x, d = (torch.randn(259, hidden, generator=gen).to(dtype).cuda() for _ in range(2))
    gain = torch.randn(hidden, generator=gen).to(dtype).cuda()
    total = (x.float() + d.float()).to(dtype) if add else x.clone()
    got = ops.rmsnorm(x, gain, 1e-6, delta=d if add else None).double()
    assert torch.equal(x, total)
    t = total.double()
    want = t / torch.sqrt((t * t).mean(dim=-1, keepdim=True) + 1e-6) * gain.double()
    # (bfloat16: the normed value is rounded, then its product with the gain)
    bound = 2.01 * HALF_STEP if dtype == BF else 2.0 ** -20
    assert bool(((got - want).abs() <= bound * want.abs()).all())


@pytest.mark.parametrize("dtype,hidden,rows", [(torch.bfloat16, 4096, 2369), (torch.bfloat16, 3072, 4737), (torch.float32, 512, 4737), (torch.float32, 2048, 2369)])
@pytest.mark.parametrize("add", [False, True])
def test_norms_of_more_rows_than_are_kept_have_the_same_bits(dtype, hidden, rows, add):
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(rows)
    x, d = (torch.randn(rows, hidden, generator=gen).to(dtype).cuda() for _ in range(2))
    gain = torch.rand(hidden, generator=gen).to(dtype).cuda() + 0.5
    few, many = x[1:].clone(), x.clone()
    want = ops.rmsnorm(few, gain, 1e-6, delta=d[1:] if add else None)         # a row less: the last step whose rows are kept
    assert torch.equal(ops.rmsnorm(many, gain, 1e-6, delta=d if add else None)[1:], want)
    assert torch.equal(many[1:], few)


@pytest.mark.parametrize("d", [32, 128])
def test_rotation_has_the_bits_of_rounded_float_products(d):
    """Without a norm every step is a product or a sum of two bfloat16 values: equal to float operations rounded one by one, for
    values of very different sizes."""
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(d)
    heads, kv, n = 3, 2, 70
    qkv = torch.randn(n, (heads + 2 * kv) * d, generator=gen) * 2.0 ** torch.randint(-40, 40, (n, (heads + 2 * kv) * d), generator=gen)
    qkv = qkv.to(BF).cuda()
    angle = torch.rand(n, d // 2, generator=gen) * 7
    cos, sin = angle.cos().cuda(), angle.sin().cuda()
    k_store, v_store = (torch.zeros(2, kv, 64, d, dtype=BF, device="cuda") for _ in range(2))
    pos, slot, table = ints(list(range(n))), ints([0] * n), ints([[1, 0]])
    q = ops.qk_norm_rope_store(qkv, heads, kv, d, None, None, 0.0, cos, sin, pos, slot, table, k_store, v_store)
    x = qkv.view(n, -1, d)[:, :heads + kv].float()
    lo, hi = x[..., :d // 2], x[..., d // 2:]
    c, s = cos.to(BF).float()[:, None], sin.to(BF).float()[:, None]
    r = lambda v: v.to(BF).float()
    want = torch.cat([r(r(lo * c) + r(-hi * s)), r(r(hi * c) + r(lo * s))], dim=-1).to(BF)
    assert torch.equal(q.view(n, heads, d), want[:, :heads])
    rows = torch.stack([k_store[1 - i // 64, :, i % 64] for i in range(n)])
    assert torch.equal(rows, want[:, heads:])


@pytest.mark.parametrize("gain_dtype", [BF, torch.float32])
def test_head_norm_gains_of_any_alignment(gain_dtype):
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(5)
    heads, kv, d, n = 4, 2, 128, 9
    qkv = torch.randn(n, (heads + 2 * kv) * d, generator=gen).to(BF).cuda()
    gains = torch.randn(2, d + 1, generator=gen).to(gain_dtype).cuda()
    angle = torch.rand(n, d // 2, generator=gen).cuda()
    got = []
    for qg, kg in ((gains[0, 1:], gains[1, 1:]), (gains[0, 1:].clone(), gains[1, 1:].clone())):
        stores = [torch.zeros(1, kv, 64, d, dtype=BF, device="cuda") for _ in range(2)]
        q = ops.qk_norm_rope_store(qkv, heads, kv, d, qg, kg, 1e-6, angle.cos(), angle.sin(), ints(list(range(n))), ints([0] * n),
                                   ints([[0]]), *stores)
        got.append([q, *stores])
    assert all(torch.equal(a, b) for a, b in zip(*got))


# enough blocks for 16 tokens a thread; taps whose address is no multiple of 16 bytes take the general kernel
@pytest.mark.parametrize("taps", [1, 2, 3, 4])
@pytest.mark.parametrize("aligned", [True, False])
def test_short_convolution_of_long_prompts(taps, aligned):
    from starter_b200 import ops

    gen, sizes, channels = torch.Generator().manual_seed(taps), [600, 1, 17, 16], 4100
    starts = [sum(sizes[:i]) for i in range(4)]
    x = torch.randn(sum(sizes), channels, generator=gen).to(BF).cuda()
    w = torch.randn(channels * taps + 4, generator=gen).cuda()
    w = w[4 if aligned else 1:][:channels * taps].view(channels, taps)
    bias = torch.randn(channels, generator=gen).cuda()
    state = torch.randn(4, (taps - 1) * channels, generator=gen).cuda() if taps > 1 else None
    before = state.clone() if taps > 1 else None
    out = ops.short_conv(x, 0, channels, w, bias, None, state, 0, ints([3, 0, 1, 2]), ints(starts), ints(sizes), max(sizes), "silu")
    for slot, start, size in zip([3, 0, 1, 2], starts, sizes):
        front = before[slot].view(taps - 1, channels).flip(0).double() if taps > 1 else x.new_zeros(0, channels).double()
        xs = torch.cat([front, x[start:start + size].double()])
        want, scale = bias.double().expand(size, -1).clone(), bias.double().abs().expand(size, -1).clone()
        for back in range(taps):
            term = w[:, taps - 1 - back].double() * xs[taps - 1 - back:taps - 1 - back + size]
            want, scale = want + term, scale + term.abs()
        want = want * torch.sigmoid(want)
        assert bool(((out[start:start + size].double() - want).abs() <= HALF_STEP * want.abs() + 2.0 ** -20 * scale).all())
        if taps > 1:
            assert torch.equal(state[slot].view(taps - 1, channels).flip(0).double(), xs[-(taps - 1):])


# pieces of eight (interleaved, all entries turn, every address on 16 bytes) and what goes through the general kernel
@pytest.mark.parametrize("rot, dims, dim, rank", [(64, 64, 128, 512), (64, 64, 128, 128), (16, 16, 24, 40), (64, 32, 128, 256), (24, 24, 20, 36)])
@pytest.mark.parametrize("n", [1, 67])
def test_rotated_queries_in_pieces(rot, dims, dim, rank, n):
    from starter_b200 import ops
    from starter_b200.config import InterleavedRopeSpec
    from starter_b200.parts import InterleavedRotaryTable

    gen, heads = torch.Generator().manual_seed(rot + n), 5
    tables = InterleavedRotaryTable(InterleavedRopeSpec(dims=dims, base=100.0), BF, "cuda")
    tables.ensure(100)
    cos, sin = ops.latent_tables(tables.rotation(), dims)
    q = torch.randn(n, heads * (dim + rot), generator=gen).to(BF).cuda()
    qa = torch.zeros(n, heads, rank + rot, dtype=BF, device="cuda")
    pos = ints(torch.randint(0, 100, (n,), generator=gen).tolist())
    ops.latent_rotate_q(q, qa, cos, sin, pos, heads, dim, rot, dims, rank)
    src = q.view(n, heads, dim + rot)[..., dim:].double()
    c, s = cos[pos.long(), :dims // 2].double()[:, None], sin[pos.long(), :dims // 2].double()[:, None]
    want = src.clone()
    want[..., 0:dims:2], want[..., 1:dims:2] = src[..., 0:dims:2] * c - src[..., 1:dims:2] * s, src[..., 1:dims:2] * c + src[..., 0:dims:2] * s
    assert bool(((qa[..., rank:].double() - want).abs() <= HALF_STEP * want.abs() + 2.0 ** -22 * src.abs().max()).all())
    assert not bool(qa[..., :rank].any())


# the layer's own kernels on one side: queries turned beside the gathering and the gate in the attention's last step, with the keys of a
# block of queries whole and in parts; on the other the turn and the gate by themselves
@pytest.mark.parametrize("past, new, parts", [(0, 300, 1), (1200, 130, 4)])
@pytest.mark.parametrize("sink", [True, False])
def test_latent_prompt_turns_and_gates(past, new, parts, sink, monkeypatch):
    from starter_b200 import ops
    from starter_b200.cache import SequenceCache
    from starter_b200.config import InterleavedRopeSpec
    from starter_b200.engine import StepContext, StepEntry, plan_step
    from starter_b200.engine.batch import upload
    from starter_b200.cache.layout import KVNeed
    from starter_b200.parts import InterleavedRotaryTable

    heads, dim, rot, vdim, rank = 4, 128, 64, 128, 256
    gen = torch.Generator().manual_seed(new)
    rand = lambda *shape: torch.randn(*shape, generator=gen).cuda()
    cache = SequenceCache({0: KVNeed(1, rank + rot, None, 0)}, {0: None}, past + new + 64, 1, BF, "cuda")
    slot = cache.open_sequence()
    cache.reserve(slot, past + new)
    cache.lengths[slot] = past
    arrays = plan_step([StepEntry(slot, [0] * new, [])], [past])
    cache.sync_table()
    dev = upload(arrays, torch.device("cuda:0"))
    ctx = StepContext(n_tokens=new, n_seqs=1, max_q_len=new, max_kv_len=past + new, cache=cache, host=arrays,
                      status=torch.zeros(1, dtype=torch.int32, device="cuda"),
                      **{k: dev[k] for k in ("tokens", "tok_pos", "tok_slot", "seq_slot", "seq_q_start", "seq_q_len", "seq_kv_len", "want_rows",
                                             "tile_seq", "tile_first", "block_seq", "block_first")})
    store, _ = cache.entry_pages(0)
    store.copy_(rand(*store.shape).to(BF))
    tables = InterleavedRotaryTable(InterleavedRopeSpec(dims=rot, base=100.0), BF, "cuda")
    tables.ensure(past + new)
    cos, sin = ops.latent_tables(tables.rotation(), rot)
    q, ukv = rand(new, heads * (dim + rot)).to(BF), (rand(heads * (dim + vdim), rank) * rank ** -0.5).to(BF)
    wide, sinks = (rand(new, 24 + heads * vdim) * 4).to(BF), rand(heads) if sink else None
    assert ops.prompt_splits(heads * ctx.block_first.shape[0], ctx.max_kv_len) == parts
    other = q.clone()
    args = (ukv, store, cache.block_table, ctx, heads, dim, vdim, rank, rot, 192 ** -0.5, None, sinks)
    turn = (cos, sin, ctx.tok_pos, rot, "interleaved")
    got = ops.latent_attention_prompt(q, *args, turn=turn, gate=(wide, 16)).double()
    ops.latent_rotate_q(other, other.view(new, heads, -1), cos, sin, ctx.tok_pos, heads, dim, rot, rot, dim)
    assert torch.equal(q, other)
    plain = ops.latent_attention_prompt(other, *args).double()
    want = plain * torch.sigmoid(wide[:, 16:16 + heads * vdim].double())
    # (the plain result is rounded to 8 bits, the gated one once more)
    assert bool(((got - want).abs() <= 2.01 * HALF_STEP * want.abs() + 1e-7).all())
    off = ops.latent_attention_prompt(other, *args, gate=(wide, 12)).double()        # (not on 16 bytes: a kernel of its own)
    want = plain * torch.sigmoid(wide[:, 12:12 + heads * vdim].double())
    assert bool(((off - want).abs() <= 2.01 * HALF_STEP * want.abs() + 1e-7).all())
