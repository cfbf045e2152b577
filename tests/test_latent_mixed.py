"""Latent prompts whose longer blocks are shared by two CTAs of a cluster while the shorter ones go to one each: the kernel against a CTA a
block, and the rule that says from how many steps on."""

import random
import time

import pytest
import torch

BF = torch.bfloat16


# (blocks of 1 to 20 steps, 1 to 7 in the window: every line between them, and one behind the longest; an odd number of heads leaves a CTA of a
# cluster idle; keys of 64 with values of 128 take a CTA a block whatever is asked for)
@pytest.mark.gpu
@pytest.mark.parametrize("heads", [1, 3, 4])
@pytest.mark.parametrize("dim,vdim,window,gated", [(128, 128, None, True), (64, 64, 150, False), (128, 64, None, False), (64, 128, None, False)])
def test_long_blocks_in_two_parts_short_ones_whole(heads, dim, vdim, window, gated, monkeypatch):
    from starter_b200 import ops
    from test_gpu_key_parts import LENGTHS, PAST, step

    rank = 128
    steps = ops.latent_block_steps([p + n for p, n in zip(PAST, LENGTHS)], LENGTHS, window)
    assert len(set(steps)) > 4
    gen, table, (rows, _), ctx = step(1, rank + 64, 16, heads)
    q = torch.randn(sum(LENGTHS), heads * (dim + 64), generator=gen).to(BF).cuda()
    ukv = (torch.randn(heads * (dim + vdim), rank, generator=gen) * rank ** -0.5).to(BF).cuda()
    gate = (torch.randn(sum(LENGTHS), heads * vdim, generator=gen).to(BF).cuda(), 0) if gated else None
    sink = torch.linspace(-1.0, 2.0, heads).cuda()

    def run(splits):
        monkeypatch.setattr(ops, "prompt_splits", lambda *a, **k: splits)
        return ops.latent_attention_prompt(q, ukv, rows, table, ctx, heads, dim, vdim, rank, 64, (dim + 64) ** -0.5, window, sink, gate=gate)

    whole = run(1)
    for split_from in sorted(set(steps)) + [steps[0] + 1]:
        got = run(2 | split_from << 8)
        assert torch.equal(got, whole) == (split_from > steps[0] or (dim, vdim) == (64, 128))
        # (the parts' sums join in another order: a rounding to 8 bits that falls on the other side)
        assert float((got.float() - whole.float()).abs().max()) <= 2.0 ** -7 * float(whole.float().abs().max())
    assert int(ctx.status.item()) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("heads,new,past,window,split_from", [(16, [1300], [0], None, 16), (16, [1300], [700], 1500, 25), (5, [2048, 1700], [0, 0], None, 8)])
def test_a_steps_own_plan_reaches_the_kernel(heads, new, past, window, split_from, monkeypatch):
    import test_gpu_key_parts as parts
    from starter_b200 import ops

    monkeypatch.setattr(parts, "LENGTHS", new)
    monkeypatch.setattr(parts, "PAST", past)
    rank, dim = 64, 128
    gen, table, (rows, _), ctx = parts.step(1, rank + 64, 16, heads)
    q = torch.randn(sum(new), heads * (dim + 64), generator=gen).to(BF).cuda()
    ukv = (torch.randn(heads * 2 * dim, rank, generator=gen) * rank ** -0.5).to(BF).cuda()
    lib, asked = ops._lib("attention_latent_prompt"), []
    entry = lib.sb_latent_prompt
    monkeypatch.setattr(lib, "sb_latent_prompt", lambda *a: (asked.append(a[-4]), entry(*a))[1])
    run = lambda: ops.latent_attention_prompt(q, ukv, rows, table, ctx, heads, dim, dim, rank, 64, 192 ** -0.5, window)
    got = run().float()
    monkeypatch.setattr(ops, "latent_mixed_splits", lambda *a: 1)
    whole = run().float()
    assert asked == [2 | split_from << 8, 1] and int(ctx.status.item()) == 0
    assert float((got - whole).abs().max()) <= 2.0 ** -7 * float(whole.abs().max()) and not torch.equal(got, whole)


@pytest.mark.parametrize("window", [None, 1, 64, 300])
def test_steps_of_blocks(window):
    from starter_b200 import ops

    kv, new = [700, 257, 64, 1500], [700, 1, 64, 513]
    want = []
    for k, n in zip(kv, new):
        sees = [range(max(0, p - window + 1) if window else 0, p + 1) for p in range(k - n, k)]
        for first in range(0, n, 256):
            keys = {key for s in sees[first:first + 256] for key in s}
            want.append(len({(key - sees[0][0]) // 64 for key in keys}))
    assert ops.latent_block_steps(kv, new, window) == tuple(sorted(want, reverse=True))


def test_which_blocks_are_shared():
    from starter_b200 import ops

    # a causal prompt's last blocks; blocks of one length, and one that two CTAs could not end before: none
    assert ops.latent_mixed_splits((32, 28, 24, 20, 16, 12, 8, 4), 16) == 2 | 28 << 8
    assert ops.latent_mixed_splits((25, 24, 20, 16, 12, 8, 4), 16) == 2 | 24 << 8
    assert ops.latent_mixed_splits((38, 35, 31, 27, 23), 16) == 2 | 27 << 8
    assert ops.latent_mixed_splits((20, 20, 20, 20, 16, 12, 8, 4), 16) == 1
    assert ops.latent_mixed_splits((16, 16, 12, 12, 8, 8, 4, 4), 16) == 1
    assert ops.latent_mixed_splits((10,), 100) == 1
    for heads in (1, 2, 40, 75, 148):
        for steps in ((1,), (500,), (60, 3), (60, 60)):
            got = ops.latent_mixed_splits(steps, heads)
            assert got == 1 or (got & 255 == 2 and 1 <= got >> 8 <= steps[0])


def test_the_plan_is_the_estimates_least():
    from starter_b200 import ops

    def plain(steps, heads):
        def cost(split_from):
            jobs = sorted((job for s in steps for job in (2 * [-(-s // 2) + 9] if s >= split_from else [s + 3]) * heads), reverse=True)
            behind = [jobs[147 - i] + jobs[148 + i] + 10 for i in range(min(148, len(jobs) - 148))]
            return max([jobs[0]] + behind), split_from
        most, split_from = min(cost(s) for s in set(steps))
        return 2 | split_from << 8 if most <= 0.93 * (max(steps) + 3) else 1

    rng, shared = random.Random(1), 0
    for _ in range(400):
        heads = rng.choice((1, 2, 5, 12, 16))
        lengths = [rng.randint(1, 80) for _ in range(rng.randint(1, 16))]
        steps = tuple(sorted((rng.choice(lengths) for _ in range(rng.randint(75 // heads + 1, 148 // heads))), reverse=True))
        shared += plain(steps, heads) > 1
        assert ops.latent_mixed_splits(steps, heads) == plain(steps, heads)
    assert 50 < shared < 350
    assert ops.latent_mixed_splits((), 4) == ops.latent_mixed_splits((5, 0), 4) == ops.latent_mixed_splits((5, -2, -7), 100) == 1
    with pytest.raises(TypeError):
        ops.latent_mixed_splits(("a",), 4)


@pytest.mark.parametrize("heads,tokens", [(16, 2048), (4, 7000), (1, 36000)])
def test_a_plan_for_new_lengths_costs_little(heads, tokens):
    """(It stands in front of the launches of a step's first latent layer, whose gain is some 10 us.)"""
    from starter_b200 import ops

    took = []
    for i in range(7):
        began = time.perf_counter()
        ops.latent_mixed_splits(ops.latent_block_steps([tokens + i], [tokens + i], None), heads)
        took.append(time.perf_counter() - began)
    assert min(took[1:]) < 1e-4
