"""The matrix-state recurrences' kernels for many tokens a sequence: against the plain statements, against the kernel
for few tokens, across the edges of their blocks of 16 (and 8) tokens and of their columns, the state carried."""

import pytest
import torch

import plain_bavedra as bavedra
import plain_salulorn as salulorn
import plain_setotar as setotar

pytestmark = pytest.mark.gpu
F = torch.float64
BF = torch.bfloat16


def packed(lengths, slots):
    starts = [sum(lengths[:i]) for i in range(len(lengths))]
    return tuple(torch.tensor(x, dtype=torch.int32).cuda() for x in (slots, starts, lengths))


def stated(mode, q, k, v, a, b, A, bias, skip, decay, heads, groups, n, width):
    """One sequence from an empty state, in float64."""
    t = q.shape[0]
    q, k, v = q.reshape(t, groups, n), k.reshape(t, groups, n), v.reshape(t, heads, width)
    if mode == "state_space":
        return bavedra.state_space_recurrence(v, k, q, bavedra.softplus(a + bias), A, skip)
    if mode == "gated_delta":
        g = torch.exp(-torch.exp(A) * bavedra.softplus(a + bias))
        return bavedra.delta_recurrence(bavedra.unit(q) * n ** -0.5, bavedra.unit(k), v, torch.sigmoid(b), g)
    if mode == "forget_write":
        low = A.reshape(heads, n)
        f = low + (1.0 - low) * torch.sigmoid(k + bias.reshape(heads, n))
        return setotar.forget_recurrence(setotar.silu(q), f, v)
    return salulorn.decayed_recurrence(q * n ** -0.5, k, v, 1.0 - decay.reshape(t, heads, n))


def form(mode, monkeypatch):
    """The mode; "segments" is a state-space step that is not walked at once, whatever its size."""
    from starter_b200 import ops

    if mode == "segments":
        monkeypatch.setattr(ops, "scan_one_walk", lambda *a: False)
        return "state_space"
    if mode == "state_space":
        monkeypatch.setattr(ops, "scan_one_walk", lambda *a: True)
    return mode


@pytest.mark.parametrize("mode", ["state_space", "segments", "gated_delta", "forget_write", "channel_decay"])
@pytest.mark.parametrize("heads,groups,n,width", [(2, 1, 128, 64), (4, 2, 72, 24), (10, 1, 104, 8), (3, 3, 120, 40)])
def test_many_tokens_a_sequence(mode, heads, groups, n, width, monkeypatch):
    from starter_b200 import ops

    mode = form(mode, monkeypatch)
    if mode in ("forget_write", "channel_decay"):
        groups = heads
    gen = torch.Generator().manual_seed(heads * n)
    lengths, slots = [129, 64, 72, 135], [2, 0, 3, 1]
    total = sum(lengths)

    def rows(columns, scale=1.0):
        return (torch.randn(total, columns, generator=gen, dtype=F) * scale).to(BF).cuda()

    # (queries and keys as columns of one tensor, in front of them columns that are not read)
    qk = rows(8 + 2 * groups * n, 0.7)
    v, ab = rows(heads * width), rows(2 * heads)
    per = heads * n if mode == "forget_write" else heads
    A = torch.linspace(0.0, 0.95, per) if mode == "forget_write" else torch.linspace(-8.0, 0.5, per)
    bias, skip = torch.randn(per, generator=gen) * 0.5, torch.linspace(-1.0, 2.0, heads)
    decay = None
    if mode == "channel_decay":
        decay = (1.0 - torch.sigmoid(torch.randn(total, heads * n, generator=gen, dtype=F) * 3.0) ** (1 / 16)).float()
    state = torch.zeros(4, 3 + heads * n * width, device="cuda")
    scalars = mode in ("state_space", "gated_delta")

    def run(pick, lens, sl):
        p, vv, raw = qk[pick].contiguous(), v[pick].contiguous(), ab[pick].contiguous()
        return ops.state_scan(
            mode, (p, 8), (p, 8 + groups * n), (vv, 0), (raw, 0) if scalars else None, (raw, heads) if mode == "gated_delta" else None,
            None if decay is not None else A.cuda(), None if decay is not None else bias.cuda(),
            skip.cuda() if mode == "state_space" else None, state, 3, *packed(lens, sl), heads, groups, n, width,
            decay=decay[pick.cpu()].cuda().contiguous() if decay is not None else None)

    assert ops._lib("state_scan_prompt").sb_scan_prompt_floats(
        1, ops.SCAN_MODES[mode], ops._at(qk, 8), qk.shape[1], ops._at(qk, 8 + groups * n), qk.shape[1], v, v.shape[1],
        None, heads, groups, n, width) >= 0
    everything = torch.arange(total).cuda()
    got = run(everything, lengths, slots)
    kept = state.clone()
    want, at = [], 0
    host = [x.double().cpu() for x in (qk[:, 8:8 + groups * n], qk[:, 8 + groups * n:], v, ab[:, :heads], ab[:, heads:])]
    for length in lengths:
        part = slice(at, at + length)
        want.append(stated(mode, *(x[part] for x in host), A.double(), bias.double(), skip.double(),
                           decay[part].double() if decay is not None else None, heads, groups, n, width))
        at += length
    want = torch.cat(want).reshape(total, heads * width)
    # float arithmetic on exact inputs: sums of up to 128 products in chains over up to 135 tokens
    assert float((got.cpu().double() - want).abs().max()) <= 2e-5 * float(want.abs().max())
    # the same by the kernel for few tokens
    state.zero_()
    monkeypatch.setattr(ops, "SCAN_PROMPT_TOKENS", 1 << 30)
    few = run(everything, lengths, slots)
    assert float((got - few).abs().max()) <= 2e-5 * float(few.abs().max())
    assert float((kept - state).abs().max()) <= 2e-5 * float(state.abs().max())
    # and in two portions
    monkeypatch.setattr(ops, "SCAN_PROMPT_TOKENS", 1)
    state.zero_()
    out = torch.empty_like(got)
    starts = [sum(lengths[:i]) for i in range(4)]
    for sizes, done in (([61, 1, 16, 130], [0, 0, 0, 0]), ([68, 63, 56, 5], [61, 1, 16, 130])):
        pick = torch.cat([torch.arange(s + d, s + d + m) for s, d, m in zip(starts, done, sizes)]).cuda()
        out[pick] = run(pick, sizes, slots)
    assert float((out - got).abs().max()) <= 2e-5 * float(got.abs().max())
    assert float((kept - state).abs().max()) <= 2e-5 * float(state.abs().max())


@pytest.mark.parametrize("mode", ["state_space", "segments", "gated_delta", "forget_write", "channel_decay"])
@pytest.mark.parametrize("which", ["q", "k", "v"])
def test_a_token_that_is_not_finite_leaves_earlier_tokens_alone(mode, which, monkeypatch):
    from starter_b200 import ops

    mode = form(mode, monkeypatch)
    heads, n, width, tokens, bad = 2, 128, 32, 70, 37
    gen = torch.Generator().manual_seed(heads + n)
    ins = {name: torch.randn(tokens, heads * size, generator=gen).to(BF).cuda()
           for name, size in (("q", n), ("k", n), ("v", width), ("ab", 2))}
    per = heads * n if mode == "forget_write" else heads
    A, bias, skip = torch.linspace(-2.0, -1.0, per).cuda(), torch.zeros(per).cuda(), torch.ones(heads).cuda()
    decay = torch.full((tokens, heads * n), 0.1).cuda() if mode == "channel_decay" else None
    scalars = mode in ("state_space", "gated_delta")

    def run():
        state = torch.zeros(1, heads * n * width, device="cuda")
        return ops.state_scan(
            mode, (ins["q"], 0), (ins["k"], 0), (ins["v"], 0), (ins["ab"], 0) if scalars else None,
            (ins["ab"], heads) if mode == "gated_delta" else None, None if decay is not None else A.sigmoid(),
            None if decay is not None else bias, skip if mode == "state_space" else None, state, 0, *packed([tokens], [0]), heads,
            heads, n, width, decay=decay)

    want = run()
    ins[which][bad, 3] = float("inf")
    got = run()
    assert torch.equal(got[:bad], want[:bad])
    # (forget-write's keys are gates: an infinite one is an open gate)
    assert bool(got[bad].isfinite().all()) == (mode == "forget_write" and which == "k")


@pytest.mark.parametrize("mode", ["state_space", "segments", "gated_delta", "forget_write", "channel_decay"])
def test_more_tokens_than_a_grid_counts_in_its_second_dimension(mode, monkeypatch):
    from starter_b200 import ops

    mode = form(mode, monkeypatch)
    heads, n, width, lengths = 1, 72, 8, [33000, 32600]
    total, gen = sum(lengths), torch.Generator().manual_seed(9)
    q, k, v, ab = (torch.randn(total, size, generator=gen).to(BF).cuda() for size in (n, n, width, 8))
    per = n if mode == "forget_write" else 1
    A, bias = torch.full((per,), 0.3).cuda(), torch.zeros(per).cuda()
    decay = torch.full((total, n), 0.1).cuda() if mode == "channel_decay" else None
    scalars, outs = mode in ("state_space", "gated_delta"), []
    for tokens in (64, 1 << 30):
        monkeypatch.setattr(ops, "SCAN_PROMPT_TOKENS", tokens)
        state = torch.zeros(2, n * width, device="cuda")
        out = ops.state_scan(
            mode, (q, 0), (k, 0), (v, 0), (ab, 0) if scalars else None, (ab, 1) if mode == "gated_delta" else None,
            None if decay is not None else A, None if decay is not None else bias, bias if mode == "state_space" else None, state, 0,
            *packed(lengths, [1, 0]), heads, heads, n, width, decay=decay)
        outs.append((out, state))
    for got, want in zip(*outs):
        # (the bound of the comparison above: the state forgets within some ten tokens)
        assert float((got - want).abs().max()) <= 2e-5 * float(want.abs().max())


@pytest.mark.parametrize("mode, floats", [("state_space", 20), ("gated_delta", 36), ("forget_write", 2 * 72)])
def test_scratch_is_bounded(mode, floats, monkeypatch):
    """A step whose scratch would take more bytes than are allowed is served by the kernel for few tokens."""
    from starter_b200 import ops

    heads, n, width, tokens = 2, 72, 8, 70
    gen = torch.Generator().manual_seed(4)
    q, k, v, ab = (torch.randn(tokens, heads * size, generator=gen).to(BF).cuda() for size in (n, n, width, 2))
    per = heads * n if mode == "forget_write" else heads
    A, bias = torch.full((per,), 0.3).cuda(), torch.zeros(per).cuda()

    def run():
        state = torch.zeros(1, heads * n * width, device="cuda")
        return ops.state_scan(mode, (q, 0), (k, 0), (v, 0), (ab, 0) if mode != "forget_write" else None,
                              (ab, heads) if mode == "gated_delta" else None, A, bias, bias if mode == "state_space" else None, state, 0,
                              *packed([tokens], [0]), heads, heads, n, width)

    many = run()
    monkeypatch.setattr(ops, "SCAN_PROMPT_BYTES", 4 * floats * heads * tokens)
    assert torch.equal(run(), many)
    monkeypatch.setattr(ops, "SCAN_PROMPT_BYTES", 4 * floats * heads * tokens - 1)
    few = run()
    monkeypatch.setattr(ops, "SCAN_PROMPT_TOKENS", 1 << 30)
    assert torch.equal(few, run()) and not torch.equal(few, many)


@pytest.mark.parametrize("segs", [2, 3, 7, 16])
@pytest.mark.parametrize("width", [64, 72])
def test_state_space_in_segments(segs, width, monkeypatch):
    """Sequences cut into segments that are walked at once, some with fewer blocks of 16 tokens than segments, against one walk."""
    from starter_b200 import ops

    heads, n = 3, 72
    gen = torch.Generator().manual_seed(segs)
    lengths, slots = [1, 16, 17, 113, 240, 400], [5, 0, 3, 1, 2, 4]
    total = sum(lengths)
    qk, v, ab = (torch.randn(total, size, generator=gen).to(BF).cuda() for size in (2 * n, heads * width, heads))
    A, bias, skip = torch.linspace(-6.0, 0.5, heads).cuda(), torch.zeros(heads).cuda(), torch.ones(heads).cuda()
    start = torch.randn(6, heads * n * width, generator=gen).cuda()

    def run(count):
        monkeypatch.setattr(ops, "scan_one_walk", lambda *a: count == 0)
        monkeypatch.setattr(ops, "scan_segments", lambda *a: count)
        state = start.clone()
        out = ops.state_scan("state_space", (qk, n), (qk, 0), (v, 0), (ab, 0), None, A, bias, skip, state, 0, *packed(lengths, slots),
                             heads, 1, n, width)
        return out, state

    (got, state), others = run(segs), (run(0), run(1))
    # float arithmetic in another order: some hundred roundings of 2^-24 of terms that may cancel
    for want, kept in others:
        assert float((got - want).abs().max()) <= 2e-5 * float(want.abs().max())
        assert float((state - kept).abs().max()) <= 2e-5 * float(kept.abs().max())


def test_segments_of_a_step():
    from starter_b200 import ops

    for tokens, seqs, blocks in ((64, 1, 32), (2048, 1, 32), (300, 1, 1), (5, 3, 8), (1 << 20, 4, 1), (40000, 600, 32)):
        segs = ops.scan_segments(tokens, seqs, blocks)
        assert 1 <= segs <= 16 and (segs == 1 or (segs * seqs * blocks <= 2 * 148 and tokens // seqs >= 48 * segs))
    # one walk where sequences are short, or its blocks fill the SMs evenly and segments are few
    for tokens, seqs, blocks, once in ((64, 1, 16, True), (191, 1, 16, True), (192, 1, 16, False), (2048, 1, 32, False), (286, 2, 24, True),
                                       (288, 2, 24, False), (2000, 4, 16, True), (2800, 4, 16, False), (8000, 4, 24, True),
                                       (64 * 7, 7, 16, False), (64, 1, 111, True), (64, 1, 112, False)):
        assert ops.scan_one_walk(tokens, seqs, blocks) is once


@pytest.mark.parametrize("segs", [2, 4])
def test_what_segments_leave_of_a_state(segs, monkeypatch):
    """Segments that keep a ten-thousandth of what they find and write nothing: what is left is as exact as its exponent."""
    from starter_b200 import ops

    heads, n, width, tokens = 2, 72, 24, 110 * segs
    gen = torch.Generator().manual_seed(segs)
    qk = torch.randn(tokens, 2 * n, generator=gen).to(BF).cuda()
    v, raw = torch.zeros(tokens, heads * width, dtype=BF).cuda(), (torch.rand(tokens, heads, generator=gen) - 2.2).to(BF).cuda()
    A, bias = torch.tensor([-0.5, -0.6]), torch.zeros(heads)
    start = torch.randn(1, heads * n * width, generator=gen).cuda()
    monkeypatch.setattr(ops, "scan_one_walk", lambda *a: False)
    monkeypatch.setattr(ops, "scan_segments", lambda *a: segs)
    state = start.clone()
    ops.state_scan("state_space", (qk, n), (qk, 0), (v, 0), (raw, 0), None, A.cuda(), bias.cuda(), None, state, 0, *packed([tokens], [0]),
                   heads, 1, n, width)
    x = A.to(F).exp() * bavedra.softplus(raw.cpu().to(F)).sum(dim=0)
    assert 6.0 * segs < float(x.min()) < float(x.max()) < 14.0 * segs
    left = state.cpu().to(F).view(heads, -1) / start.cpu().to(F).view(heads, -1) * x.exp()[:, None]
    # the exponent's factors and their product round by up to 2^-23 of it each; the last segment's eight blocks, which keep a
    # quarter, by 2^-23 of what they keep
    assert float((left - 1.0).abs().max()) <= (3.0 * float(x.max()) + 8 * 4) * 2.0 ** -23
