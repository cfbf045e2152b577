"""Latent attention of single tokens with up to 16 heads against 64 bits: lengths around a page, windows that begin inside one, parts of which
some are empty, latents that leave some of a block's warps without columns, and rows whose last step of sixteen entries stands alone."""

import pytest
import torch

pytestmark = pytest.mark.gpu
BF, F = torch.bfloat16, torch.float64


@pytest.mark.parametrize("heads, rank, rot", [(16, 512, 64), (5, 256, 64), (1, 16, 16), (16, 272, 48), (8, 64, 32), (12, 512, 128)])
@pytest.mark.parametrize("window", [None, 1, 70, 128])
@pytest.mark.parametrize("sink", [False, True])
def test_single_tokens(heads, rank, rot, window, sink):
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(rank + heads)
    lengths, width, scale = [1, 63, 64, 65, 200, 700], rank + rot, (rank + rot) ** -0.5
    n, per = len(lengths), 11
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    table = torch.randperm(n * per, generator=gen).int().view(n, per).cuda()
    store = torch.randn(n * per, 1, 64, width, generator=gen).to(BF).cuda()
    slots = list(reversed(range(n)))
    for slot, length in zip(slots, lengths):                        # what lies behind a sequence is nobody's number
        page, at = int(table[slot, (length - 1) // 64]), (length - 1) % 64 + 1
        store[page, 0, at:] = float("nan")
    qa = torch.randn(n, heads, width, generator=gen).to(BF).cuda() * 2
    sinks = torch.randn(heads, generator=gen).cuda() if sink else None
    want = torch.empty(n, heads, rank, dtype=F, device="cuda")
    for i, (slot, length) in enumerate(zip(slots, lengths)):
        rows = torch.cat([store[int(p), 0] for p in table[slot]])[:length].to(F)
        first = max(0, length - window) if window else 0
        s = qa[i].to(F) @ rows[first:].T * scale
        if sink:
            s = torch.cat([s, sinks[:, None].to(F)], dim=1)
        want[i] = torch.softmax(s, dim=1)[:, :length - first] @ rows[first:, :rank]
    seqs = (ints(slots), ints(list(range(n))), ints([1] * n), ints(lengths), ints(list(range(n))), ints([0] * n))
    for splits in (1, 2, 5, 32):
        got = ops.latent_attention_tc(qa, store, table, *seqs, heads, rank, rot, scale, window, splits, 1, sinks).to(F)
        # (weights of at most one are rounded to 8 bits, and the result)
        assert bool(((got - want).abs() <= 2.0 ** -7.5 * (want.abs() + want.abs().amax(-1, keepdim=True))).all()), splits
        old = ops.latent_attention_tc(qa, store, table, *seqs, heads, rank, rot, scale, window, splits, 0, sinks).to(F)
        assert float((got - want).norm()) <= 1.05 * float((old - want).norm()) + 1e-6 * float(want.norm())


@pytest.mark.parametrize("window", [1, 70, 128])
@pytest.mark.parametrize("splits", [1, 3])
def test_rows_in_front_of_the_window_do_not_count(window, splits):
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(window)
    heads, rank, rot, lengths, per = 16, 256, 64, [1, 65, 129, 191, 192, 700], 11
    n, width = len(lengths), rank + rot
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    table = torch.randperm(n * per, generator=gen).int().view(n, per).cuda()
    store = torch.randn(n * per, 1, 64, width, generator=gen).to(BF).cuda()
    qa = torch.randn(n, heads, width, generator=gen).to(BF).cuda()
    seqs = (ints(list(range(n))), ints(list(range(n))), ints([1] * n), ints(lengths), ints(list(range(n))), ints([0] * n))
    run = lambda: ops.latent_attention_tc(qa, store, table, *seqs, heads, rank, rot, width ** -0.5, window, splits, 1)
    want = run()
    assert bool(torch.isfinite(want).all())
    for slot, length in enumerate(lengths):
        for at in range(max(0, length - window)):
            store[int(table[slot, at // 64]), 0, at % 64] = (float("nan"), float("inf"), -float("inf"))[at % 3]
    assert torch.equal(run(), want)


def test_parts_of_whole_pages():
    from starter_b200 import ops

    for rows in (1, 2, 8, 40, 148, 300):
        for keys in (1, 64, 65, 1000, 2048, 3073):
            for window in (None, 512, 1000):
                parts = ops.latent_splits(rows, 16, window, keys)
                pages = -(-min(window or keys, keys) // 64) + (1 if window and window < keys else 0)
                each = -(-pages // parts)
                assert 1 <= parts <= 32 and (parts == 1 or parts * rows <= 148) and each * (parts - 1) < pages
