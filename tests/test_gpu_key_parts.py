"""Prompt attention whose blocks' keys are shared by the CTAs of a cluster, against one CTA a block: plain, with every extra, over
formed keys; sequences of a few keys (fewer steps than parts), ragged ones, windows, chunks."""

from types import SimpleNamespace

import pytest
import torch

from starter_b200.engine.batch import plan_step

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
LENGTHS, PAST = [300, 1, 700, 129, 256], [0, 40, 513, 1100, 64]


def step(n_heads_kv, dim, vdim, seed):
    """Pages of random keys and values, and the step's arrays."""
    pages = [-(-(p + n) // 64) for p, n in zip(PAST, LENGTHS)]
    gen = torch.Generator().manual_seed(seed)
    table, at = torch.zeros(len(pages), max(pages), dtype=torch.int32), 0
    for i, n in enumerate(pages):
        table[i, :n] = torch.randperm(n, generator=gen) + at
        at += n
    store = [(torch.randn(at, n_heads_kv, 64, size, generator=gen)).to(BF).cuda() for size in (dim, vdim)]
    arrays = plan_step([SimpleNamespace(slot=i, tokens=[0] * n, want=[]) for i, n in enumerate(LENGTHS)], PAST)
    ctx = SimpleNamespace(host=arrays, n_seqs=len(LENGTHS), max_q_len=max(LENGTHS), max_kv_len=int(arrays["seq_kv_len"].max()),
                          status=torch.zeros(1, dtype=torch.int32).cuda(),
                          **{k: torch.from_numpy(v).cuda() for k, v in arrays.items()})
    return gen, table.cuda(), store, ctx


def same(monkeypatch, run, status):
    """Every number of parts gives what one gives, but for roundings: weights and outputs round to 2^-9 of themselves each."""
    from starter_b200 import ops

    got = {}
    for parts in (1, 2, 4):
        monkeypatch.setattr(ops, "prompt_splits", lambda *a, **k: parts)
        got[parts] = run().float()
    assert int(status.item()) == 0 and bool(torch.isfinite(got[1]).all())
    for parts in (2, 4):
        assert float((got[parts] - got[1]).abs().max()) <= 2.0 ** -7 * float(got[1].abs().max())
        assert float((got[parts] - got[1]).norm()) <= 2.0 ** -8 * float(got[1].norm())
        if parts > 2:
            assert not torch.equal(got[parts], got[1])


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("window", [None, 200])
def test_plain(dim, window, monkeypatch):
    from starter_b200 import ops

    gen, table, (keys, values), ctx = step(2, dim, dim, dim)
    q = torch.randn(sum(LENGTHS), 4 * dim, generator=gen).to(BF).cuda()
    same(monkeypatch, lambda: ops.attention_prefill(
        q, keys, values, table, ctx.seq_slot, ctx.seq_q_start, ctx.seq_q_len, ctx.seq_kv_len, ctx.tile_seq, ctx.tile_first, 4, 2, dim,
        dim ** -0.5, window, status=ctx.status, kernel="tcgen05", max_q_len=ctx.max_q_len, blocks=(ctx.block_seq, ctx.block_first),
        kv_hint=ctx.max_kv_len), ctx.status)


@pytest.mark.parametrize("dim,vdim,chunk,window,keep,cap,penalty,gated", [
    (128, 128, None, 256, 0, 50.0, False, False), (48, 40, None, None, 0, 1.0, False, True), (128, 64, 300, None, 70, None, True, True),
    (64, 64, None, 130, 5, 30.0, True, False)])
def test_with_extras(dim, vdim, chunk, window, keep, cap, penalty, gated, monkeypatch):
    from starter_b200 import ops

    gen, table, (keys, values), ctx = step(2, dim, vdim, dim + vdim)
    q = torch.randn(sum(LENGTHS), 4 * dim, generator=gen).to(BF).cuda()
    slopes = tuple(torch.rand(4, generator=gen).cuda() + 0.1 for _ in range(2)) if penalty else None
    gate = torch.rand(sum(LENGTHS), 4, generator=gen).cuda() if gated else None
    same(monkeypatch, lambda: ops.sink_attention_tcgen05(
        q, keys, values, table, ctx.seq_slot, ctx.seq_q_start, ctx.seq_q_len, ctx.seq_kv_len, ctx.tile_seq, ctx.tile_first, 4, 2, dim,
        dim ** -0.5, slopes, torch.linspace(-1.0, 2.0, 4).cuda(), gate, chunk, window, ctx.status, (ctx.block_seq, ctx.block_first), vdim,
        keep, cap, ctx.max_kv_len), ctx.status)


@pytest.mark.parametrize("dim,vdim", [(128, 128), (64, 64), (128, 64)])
@pytest.mark.parametrize("window,sink", [(None, True), (150, False)])
def test_over_formed_keys(dim, vdim, window, sink, monkeypatch):
    from starter_b200 import ops

    rank, heads = 128, 3
    gen, table, (store, _), ctx = step(1, rank + 64, 16, dim)
    q = torch.randn(sum(LENGTHS), heads * (dim + 64), generator=gen).to(BF).cuda()
    ukv = (torch.randn(heads * (dim + vdim), rank, generator=gen) * rank ** -0.5).to(BF).cuda()
    same(monkeypatch, lambda: ops.latent_attention_prompt(
        q, ukv, store, table, ctx, heads, dim, vdim, rank, 64, (dim + 64) ** -0.5, window,
        torch.linspace(-1.0, 2.0, heads).cuda() if sink else None), ctx.status)


@pytest.mark.parametrize("kind", ["plain", "window", "extras", "capped", "formed", "formed, sink"])
def test_scores_that_are_no_numbers(kind, monkeypatch):
    """A row with a score that is NaN or +infinity is no number whichever part its key lies in; every other row is what it was."""
    from starter_b200 import ops

    heads, dim, rank = 4, 128, 128
    formed = kind.startswith("formed")
    gen, table, (keys, values), ctx = step(1, rank + 64, 16, 5) if formed else step(2, dim, dim, 5)
    q = torch.randn(sum(LENGTHS), heads * (dim + 64 if formed else dim), generator=gen).to(BF).cuda()

    def key(seq, pos):
        return keys[int(table[seq, pos // 64]), :, pos % 64]

    key(2, 600)[:, -3] = float("nan")                  # (of a formed key's row the shared part, which is in no value)
    key(0, 10)[:, -5] = float("inf")                   # +infinity for about half of the queries, weight 0 for the others
    key(1, 12)[:, -1] = float("-inf")
    q[-200] = float("nan")
    ints = (table, ctx.seq_slot, ctx.seq_q_start, ctx.seq_q_len, ctx.seq_kv_len, ctx.tile_seq, ctx.tile_first)
    blocks, sink = (ctx.block_seq, ctx.block_first), torch.linspace(-1.0, 2.0, heads).cuda()
    ukv = (torch.randn(heads * 2 * dim, rank, generator=gen) * rank ** -0.5).to(BF).cuda()

    def run():
        if formed:
            return ops.latent_attention_prompt(q, ukv, keys, table, ctx, heads, dim, dim, rank, 64, (dim + 64) ** -0.5, None,
                                               sink if "sink" in kind else None)
        if kind in ("plain", "window"):
            return ops.attention_prefill(q, keys, values, *ints, heads, 2, dim, dim ** -0.5, 300 if kind == "window" else None,
                                         status=ctx.status, kernel="tcgen05", max_q_len=ctx.max_q_len, blocks=blocks,
                                         kv_hint=ctx.max_kv_len)
        return ops.sink_attention_tcgen05(q, keys, values, *ints, heads, 2, dim, dim ** -0.5, None, sink, None, None, 400, ctx.status,
                                          blocks, dim, 0, 30.0 if kind == "capped" else None, ctx.max_kv_len)

    got = {}
    for parts in (1, 2, 4):
        monkeypatch.setattr(ops, "prompt_splits", lambda *a, **k: parts)
        got[parts] = run().float()
    good = got[1].isfinite()
    # by heads: a score of +infinity is one head's (with a cap it is the cap, a number)
    by_head = good.view(sum(LENGTHS), heads, -1)
    assert torch.equal(by_head.all(2), by_head.any(2)) and not good[-200].any()
    first = 87                                          # the sequence's first query that sees the key
    last = min(LENGTHS[2], first + {"plain": 700, "window": 300}.get(kind, 700 if formed else 400))
    lost = by_head[301 + first:301 + last]
    assert not lost.any() and bool(by_head[301:301 + first].all()) and bool(by_head[301 + last:-385].all())
    assert 0.2 < float(by_head[10:300].float().mean()) < 0.9 or kind == "capped"
    for parts in (2, 4):
        assert torch.equal(got[parts].isfinite(), good)
        assert float((got[parts] - got[1])[good].abs().max()) <= 2.0 ** -7 * float(got[1][good].abs().max())


def test_parts_of_a_step():
    from starter_b200 import ops

    for blocks, keys, window, least in ((1, 5000, None, 1100), (37, 1100, None, 1100), (38, 2000, None, 1100), (74, 1100, 5000, 1100),
                                        (75, 9000, None, 1100), (10, 1099, None, 1100), (10, 5000, 512, 1100), (10, 460, 400, 450)):
        parts = ops.prompt_splits(blocks, keys, window, least)
        assert parts in (1, 2, 4) and (parts == 1 or parts * blocks <= 148)
        assert (parts > 1) == (blocks <= 74 and min(keys, window + 256 if window else keys) >= least)


def test_clusters_that_share_keys_run_at_once(monkeypatch):
    """No step gets more clusters than the device holds: those left over would walk behind the others."""
    from starter_b200 import ops

    fours, pairs = ops.prompt_clusters(4), ops.prompt_clusters(2)
    assert 1 <= fours <= 37 and fours <= pairs <= 74
    for blocks in range(1, 80):
        parts = ops.prompt_splits(blocks, 5000)
        assert parts == (4 if blocks <= fours else 2 if blocks <= pairs else 1)
    monkeypatch.setattr(ops, "prompt_clusters", lambda size: {4: 30, 2: 70}[size])
    assert [ops.prompt_splits(n, 5000) for n in (30, 31, 70, 71, 75)] == [4, 2, 2, 1, 1]


@pytest.mark.parametrize("kind", ["plain", "formed"])
@pytest.mark.parametrize("parts,left_out", [(2, 0), (4, 0), (4, 6)])
def test_a_wait_in_a_part_that_runs_out_is_reported(kind, parts, left_out, monkeypatch):
    """Values of one step are left out on purpose, which one part of a block waits for: it gives up after 2 ms, meets the others at the
    cluster's barriers, every block returns and bit 16 of the status word is set; the same call is right afterwards."""
    from starter_b200 import ops

    heads, dim, rank = 2, 128, 128
    gen, table, (keys, values), ctx = step(1, rank + 64, 16, 9) if kind == "formed" else step(1, dim, dim, 9)
    q = torch.randn(sum(LENGTHS), heads * (dim + 64 if kind == "formed" else dim), generator=gen).to(BF).cuda()
    ukv = (torch.randn(heads * 2 * dim, rank, generator=gen) * rank ** -0.5).to(BF).cuda()

    def run(withhold=None):
        if kind == "formed":
            return ops.latent_attention_prompt(q, ukv, keys, table, ctx, heads, dim, dim, rank, 64, (dim + 64) ** -0.5, None, None).float()
        return ops.attention_prefill(q, keys, values, table, ctx.seq_slot, ctx.seq_q_start, ctx.seq_q_len, ctx.seq_kv_len, ctx.tile_seq,
                                     ctx.tile_first, heads, 1, dim, dim ** -0.5, status=ctx.status, kernel="tcgen05",
                                     max_q_len=ctx.max_q_len, blocks=(ctx.block_seq, ctx.block_first), withhold=withhold,
                                     kv_hint=ctx.max_kv_len).float()

    monkeypatch.setattr(ops, "prompt_splits", lambda *a, **k: 1)
    want = run()
    monkeypatch.setattr(ops, "prompt_splits", lambda *a, **k: parts)
    if kind == "formed":
        lib = ops._lib("attention_latent_prompt")
        with monkeypatch.context() as m:
            m.setattr(lib, "sb_latent_prompt", lambda *a: lib.sb_latent_prompt_withheld(*a[:-1], left_out, 2_000_000, a[-1]))
            run()
    else:
        run((left_out, 2_000_000))
    assert ctx.status.item() == 16
    ctx.status.zero_()
    got = run()
    assert ctx.status.item() == 0 and float((got - want).abs().max()) <= 2.0 ** -7 * float(want.abs().max())
