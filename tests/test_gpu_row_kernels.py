"""Row kernels in 8- and 16-byte pieces at the widths where a thread's number of pieces changes: the norm of parts with a gate and
the latent attention's norms and rotation."""

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
HALF_STEP = 2.0 ** -8 * 1.01     # rounding to bfloat16 and a little for the sums in 32 bits


# a warp with one and two pieces a lane, a block of 128 and of 256 threads with two, four and eight pieces a thread
@pytest.mark.parametrize("psize", [4, 128, 132, 256, 260, 1024, 1028, 2052, 4096, 4100, 8192])
@pytest.mark.parametrize("order", ["gate first", "norm first", "no gate"])
def test_norm_of_parts_with_a_gate(psize, order):
    from starter_b200 import ops

    rows, parts = 5, 3 if psize < 2000 else 2
    width, gen = psize * parts, torch.Generator().manual_seed(psize)
    o = (torch.randn(rows, width, generator=gen) * 2).cuda()
    z = (torch.randn(rows, width + 8, generator=gen) * 3).to(BF).cuda()
    for gain in (torch.randn(width, generator=gen).cuda(), torch.randn(psize, generator=gen).cuda()):
        got = ops.group_norm_gate(o, None if order == "no gate" else z, 4 if order != "no gate" else 0, gain, parts, 1e-5,
                                  order == "gate first", BF).double()
        g = torch.nn.functional.silu(z[:, 4:4 + width].double())
        x = o.double() * g if order == "gate first" else o.double()
        x = x.view(rows, parts, psize)
        x = (x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + 1e-5)).flatten(1) * gain.double().repeat(width // gain.shape[0])
        want = x * g if order == "norm first" else x
        assert bool(((got - want).abs() <= HALF_STEP * want.abs()).all())


# one and two pieces of the query latent a thread; a key/value latent that reaches the warp that turns the shared part
@pytest.mark.parametrize("q_rank, rank, rot, dims", [(8, 8, 8, 8), (1536, 512, 64, 64), (2056, 256, 64, 32), (4096, 1800, 72, 72), (512, 2048, 16, 4)])
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("write", [True, False])
def test_latent_prepare_in_pieces(q_rank, rank, rot, dims, split, write):
    from starter_b200 import ops
    from starter_b200.config import InterleavedRopeSpec, PartialRopeSpec
    from starter_b200.parts import InterleavedRotaryTable, PartialRotaryTable

    gen = torch.Generator().manual_seed(q_rank + rank)
    pos, slot = [0, 63, 64, 130, 5], [1, 1, 1, 1, 0]
    n, kv_col = len(pos), q_rank + 8                     # (eight columns between the latents that are not read)
    proj = (torch.randn(n, kv_col + (rank + rot if write else 0), generator=gen) * 3).to(BF).cuda()
    qg, kg = torch.randn(q_rank, generator=gen).cuda(), torch.randn(rank, generator=gen).cuda()
    tables = PartialRotaryTable(PartialRopeSpec(dims=dims, base=100.0), BF, "cuda") if split else \
        InterleavedRotaryTable(InterleavedRopeSpec(dims=dims, base=100.0), BF, "cuda")
    tables.ensure(200)
    rotation = tables.rotation()
    cos, sin = ops.latent_tables(rotation, dims)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    table = ints([[4, 0, 0], [3, 1, 2]])
    store = torch.zeros(5, 1, 64, rank + rot, dtype=BF, device="cuda")
    cq = ops.latent_prepare(proj, qg, kg if write else None, 1e-5, cos, sin, ints(pos), ints(slot), table, store if write else None,
                            q_rank, rank, rot, dims, write_cache=write, layout=rotation.layout, kv_col=kv_col)
    p = proj.double()

    def norm(x, gain):
        return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + 1e-5) * gain.double()

    want = norm(p[:, :q_rank], qg)
    assert bool(((cq.double() - want).abs() <= HALF_STEP * want.abs()).all())
    if not write:
        return
    rows = torch.stack([store[int(table[s, q // 64]), 0, q % 64] for s, q in zip(slot, pos)]).double()
    want = norm(p[:, kv_col:kv_col + rank], kg)
    assert bool(((rows[:, :rank] - want).abs() <= HALF_STEP * want.abs()).all())
    shared = p[:, kv_col + rank:]
    one, two = (slice(0, dims // 2), slice(dims // 2, dims)) if split else (slice(0, dims, 2), slice(1, dims, 2))
    c, s = cos[ints(pos).long(), :dims // 2].double(), sin[ints(pos).long(), :dims // 2].double()
    want = shared.clone()
    want[:, one], want[:, two] = shared[:, one] * c - shared[:, two] * s, shared[:, two] * c + shared[:, one] * s
    assert bool(((rows[:, rank:] - want).abs() <= HALF_STEP * want.abs() + 2.0 ** -22 * shared.abs().max()).all())
    assert int((store.float().abs().sum(dim=-1) > 0).sum()) == n


# steps in which every sequence is listed with what it brings: whole pieces of eight tokens and rests, sequences shorter than the
# filter beside long ones, many sequences of two tokens, single tokens
@pytest.mark.parametrize("steps, channels", [([[150, 1, 9, 8], [7, 8, 2, 16], [1, 1, 1, 1]], 516), ([[2] * 130, [1] * 130, [3] * 130], 12)])
@pytest.mark.parametrize("taps", [1, 2, 3, 4])
@pytest.mark.parametrize("act", [None, "silu"])
def test_short_convolution_in_pieces(steps, channels, taps, act):
    from starter_b200 import ops

    gen, n = torch.Generator().manual_seed(channels + taps), len(steps[0])
    lengths = [sum(s[i] for s in steps) for i in range(n)]
    x = [torch.randn(length, 4 + channels + 8, generator=gen).to(BF) for length in lengths]
    w, bias, in_bias = torch.randn(channels, taps, generator=gen), torch.randn(channels, generator=gen), torch.randn(channels, generator=gen)
    slots = list(reversed(range(n)))
    state = torch.zeros(n, (taps - 1) * channels + 3, device="cuda") if taps > 1 else None
    done, got = [0] * n, [[] for _ in range(n)]
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    for sizes in steps:
        rows = torch.cat([x[i][done[i]:done[i] + m] for i, m in enumerate(sizes)]).cuda()
        starts = [sum(sizes[:i]) for i in range(n)]
        out = ops.short_conv(rows, 4, channels, w.cuda(), bias.cuda(), in_bias.cuda(), state, 3 if taps > 1 else 0, ints(slots), ints(starts), ints(sizes),
                             max(sizes), act).cpu()
        for i, m in enumerate(sizes):
            got[i].append(out[starts[i]:starts[i] + m])
            done[i] += m
    for i in range(n):
        xs = x[i][:, 4:4 + channels].double() + in_bias.double()
        want, size = bias.double().expand_as(xs).clone(), bias.double().abs().expand_as(xs).clone()
        for back in range(min(taps, lengths[i])):
            want[back:] += w[:, taps - 1 - back].double() * xs[:lengths[i] - back]
            size[back:] += (w[:, taps - 1 - back].double() * xs[:lengths[i] - back]).abs()
        if act:
            want = want * torch.sigmoid(want)
        # (the slope of silu is at most 1.1)
        assert bool(((torch.cat(got[i]).double() - want).abs() <= HALF_STEP * want.abs() + 2.0 ** -20 * size).all())
