"""The experts' grouped tcgen05 products of few rows an expert: every tile height, at experts with no row, one row, whole tiles
and a row more, widths that leave part of a weight tile and of a k-block, against the plain experts in float64; the dealing of
pairs to tiles."""

import pytest
import torch

pytestmark = pytest.mark.gpu
BF, F = torch.bfloat16, torch.float64


def plain(h, ids, weights, gate_up, down, kind, limit, inner, weigh_input):
    out = torch.zeros(h.shape[0], down.shape[1], dtype=F, device="cuda")
    for e in range(gate_up.shape[0]):
        row, place = torch.nonzero(ids == e, as_tuple=True)
        if not row.numel():
            continue
        w, by = weights[row, place].to(F)[:, None], 1.0
        if weigh_input:
            by, w = w, 1.0
        p = (h[row].to(F) @ gate_up[e].to(F).T) * by
        p = p.to(BF).to(F)                                   # the products are rounded in front of the activation
        if kind == "relu2":
            a = torch.relu(p) ** 2
        else:
            g, u = p[:, :inner], p[:, inner:]
            a = g * torch.sigmoid(g) * u if kind == "gated_silu" else (
                g.clamp(max=limit) * torch.sigmoid(1.702 * g.clamp(max=limit)) * (u.clamp(-limit, limit) + 1.0))
        out.index_add_(0, row, w * (a.to(BF).to(F) @ down[e].to(F).T).to(BF).to(F))
    return out


@pytest.mark.parametrize("rows", [16, 32, 64, 128, 256])
@pytest.mark.parametrize("kind,experts,width,inner,weigh", [
    ("gated_silu", 6, 144, 192, False), ("gated_clamped", 5, 256, 64, False), ("relu2", 7, 208, 80, False), ("gated_silu", 6, 1040, 128, True),
    ("relu2", 40, 64, 272, True)])
def test_experts_by_tile_height(rows, kind, experts, width, inner, weigh, monkeypatch):
    from starter_b200 import ops

    if weigh and rows == 256:
        pytest.skip("weights in front of the experts do not go through the prompt product below 256 rows an expert")
    gen = torch.Generator().manual_seed(rows + experts)
    # rows of the experts in turn: none, one, a tile less one, a tile, a tile and one; then whatever is left
    counts = ([0, 1, rows - 1, rows, rows + 1] + [3] * experts)[:experts]
    ids = torch.tensor([e for e, n in enumerate(counts) for _ in range(n)], dtype=torch.int32)
    ids = ids[torch.randperm(ids.numel(), generator=gen)][:, None].cuda()
    tokens = ids.shape[0]
    gated = kind != "relu2"
    h = torch.randn(tokens, width, generator=gen).to(BF).cuda()
    gate_up = (torch.randn(experts, (2 if gated else 1) * inner, width, generator=gen) * 2.0 * width ** -0.5).to(BF).cuda()
    down = (torch.randn(experts, width, inner, generator=gen) * inner ** -0.5).to(BF).cuda()
    weights = (torch.rand(tokens, 1, generator=gen) + 0.5).cuda()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    limit = 1.25 if kind == "gated_clamped" else 0.0
    monkeypatch.setattr(ops, "moe_group_rows", lambda *a: rows)
    got = ops.moe_experts(h, ids, weights, gate_up, down, limit, kind, status=status, weigh_input=weigh).double()
    want = plain(h, ids, weights, gate_up, down, kind, limit, inner, weigh)
    # a product that falls on the other side of a rounding moves by 2^-8 of itself: a rounding of each product, of the
    # activation and of the result
    scale = float(want.abs().max())
    assert int(status.item()) == 0
    assert float((got - want).abs().max()) <= 2.0 ** -6 * scale and float((got - want).norm()) <= 2.0 ** -8 * float(want.norm())


@pytest.mark.parametrize("splits", [1, 2, 4])
def test_k_range_in_parts(splits, monkeypatch):
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(splits)
    experts, width, inner, tokens = 3, 520, 128, 70
    ids = torch.randint(0, experts, (tokens, 1), generator=gen).to(torch.int32).cuda()
    h = torch.randn(tokens, width, generator=gen).to(BF).cuda()
    gate_up = (torch.randn(experts, 2 * inner, width, generator=gen) * 2.0 * width ** -0.5).to(BF).cuda()
    down = (torch.randn(experts, width, inner, generator=gen) * inner ** -0.5).to(BF).cuda()
    weights = torch.ones(tokens, 1).cuda()
    monkeypatch.setattr(ops, "moe_group_rows", lambda *a: 32)
    monkeypatch.setattr(ops, "_moe_group_plan", lambda bm, n_out, k, gated, tiles: (ops.whole_splits(-(-k // 64), splits), 4))
    got = ops.moe_experts(h, ids, weights, gate_up, down, expert="gated_silu").double()
    want = plain(h, ids, weights, gate_up, down, "gated_silu", 0.0, inner, False)
    assert float((got - want).norm()) <= 2.0 ** -8 * float(want.norm())


def test_tile_heights_of_a_step():
    from starter_b200 import ops

    for pairs, experts, weigh, rows in ((4, 16, False, 0), (96, 16, False, 0), (97, 16, False, 16), (208, 16, False, 16), (209, 16, False, 32),
                                        (448, 16, False, 32), (449, 16, False, 64), (1023, 16, False, 64), (1024, 16, False, 256),
                                        (1024, 16, True, 64), (1025, 16, True, 128), (4095, 16, True, 128), (4096, 16, True, 256)):
        assert ops.moe_group_rows(pairs, experts, weigh) == rows
        if 0 < rows < 256:
            splits, stages = ops._moe_group_plan(rows, 2048, 2048, True, min(experts, pairs))
            assert 1 <= splits <= 8 and 2 <= stages <= 8 and stages * (16384 + 128 * rows) >= 512 * rows


@pytest.mark.parametrize("pairs,experts", [(1, 1), (31, 5), (1024, 16), (1025, 16), (8191, 7), (8192, 1), (8193, 7), (20000, 130)])
def test_pairs_are_dealt_to_tiles(pairs, experts):
    """Every pair of an expert once, in that expert's tiles, and -1 behind them, where a thread's pairs are counted and placed in
    one pass (up to 8 a thread, of 256 threads up to 1,024 pairs and 1,024 beyond) and where they are walked twice."""
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(pairs)
    ids = torch.randint(0, experts + 1, (pairs,), generator=gen, dtype=torch.int32)       # (`experts`: an identity expert)
    bm = 16
    tiles = -(-pairs // bm) + min(experts, pairs)
    placed = torch.full((tiles * bm,), -7, dtype=torch.int32, device="cuda")
    tile_expert = torch.full((tiles,), -7, dtype=torch.int32, device="cuda")
    used = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops._check(ops._lib("moe").sb_moe_align(ids.cuda(), pairs, experts, placed, tiles * bm, tile_expert, used, bm, ops._stream()), "moe_align")
    placed, names, used = placed.cpu().view(tiles, bm), tile_expert.cpu(), int(used)
    counts = torch.bincount(ids, minlength=experts + 1)[:experts]
    assert used == int(((counts + bm - 1) // bm).sum())
    assert names[:used].tolist() == sorted(names[:used].tolist())
    for expert in range(experts):
        mine = placed[:used][names[:used] == expert].flatten()
        n = int(counts[expert])
        assert sorted(mine[:n].tolist()) == (ids == expert).nonzero().flatten().tolist()
        assert (mine[n:] == -1).all()


@pytest.mark.parametrize("rows,splits,stage", [(16, 1, 0), (32, 4, 1), (128, 2, 2)])
def test_a_wait_in_the_grouped_product_that_runs_out_is_reported(rows, splits, stage, monkeypatch):
    """The rows of one k-block of every block are left out on purpose (an entry point made for this): the wait on them gives up after
    2 ms, the kernel returns, bit 4 of the status word is set; the same layer without the gap is right afterwards."""
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(rows)
    experts, width, inner, tokens = 3, 1024, 768, 70
    ids = torch.randint(0, experts, (tokens, 1), generator=gen).to(torch.int32).cuda()
    h = torch.randn(tokens, width, generator=gen).to(BF).cuda()
    gate_up = (torch.randn(experts, 2 * inner, width, generator=gen) * 2.0 * width ** -0.5).to(BF).cuda()
    down = (torch.randn(experts, width, inner, generator=gen) * inner ** -0.5).to(BF).cuda()
    weights, status, lib = torch.ones(tokens, 1).cuda(), torch.zeros(1, dtype=torch.int32, device="cuda"), ops._lib("gemm_tcgen05")
    monkeypatch.setattr(ops, "moe_group_rows", lambda *a: rows)
    monkeypatch.setattr(ops, "_moe_group_plan", lambda *a: (splits, 3))

    def run():
        return ops.moe_experts(h, ids, weights, gate_up, down, expert="gated_silu", status=status).double()

    with monkeypatch.context() as m:
        m.setattr(lib, "sb_gemm_tcgen05_grouped", lambda *a: lib.sb_gemm_tcgen05_grouped_withheld(*a[:-1], 2_000_000, stage, a[-1]))
        run()
        assert status.item() == 4
    status.zero_()
    want = plain(h, ids, weights, gate_up, down, "gated_silu", 0.0, inner, False)
    assert float((run() - want).norm()) <= 2.0 ** -8 * float(want.norm()) and status.item() == 0


@pytest.mark.parametrize("tokens", [3, 70, 200])
@pytest.mark.parametrize("which", ["h", "gate_up", "down"])
def test_operands_off_their_alignment_are_refused(tokens, which):
    from starter_b200 import ops

    def made(*shape, off):
        size = 1
        for n in shape:
            size *= n
        return torch.zeros(size + 8, dtype=BF, device="cuda")[int(off):int(off) + size].view(*shape)

    h, gate_up, down = (made(*shape, off=which == name) for name, shape in (("h", (tokens, 64)), ("gate_up", (2, 128, 64)), ("down", (2, 64, 64))))
    ids, weights = torch.zeros(tokens, 1, dtype=torch.int32, device="cuda"), torch.ones(tokens, 1, device="cuda")
    with pytest.raises(ops.KernelError, match="16-byte aligned"):
        ops.moe_experts(h, ids, weights, gate_up, down, expert="gated_silu")
    assert bool((ops.moe_experts(h, ids, weights, gate_up, down, expert="gated_silu", tile_rows=32) == 0).all())


# the few-row kernel: one to eight warps a block, k ranges shorter than what its warps keep in flight, weight rows that end inside a block
@pytest.mark.parametrize("width, inner, experts, top, tokens", [(16, 16, 2, 1, 1), (48, 144, 3, 2, 5), (272, 6416, 4, 2, 3),
                                                                (1040, 2064, 16, 4, 8), (2064, 80, 8, 3, 2)])
@pytest.mark.parametrize("expert", ["gated_silu", "relu2", "gated_clamped"])
def test_few_rows_an_expert(width, inner, experts, top, tokens, expert):
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(width + inner)
    wide = inner if expert == "relu2" else 2 * inner
    h = torch.randn(tokens, width, generator=gen).to(BF).cuda()
    up = (torch.randn(experts, wide, width, generator=gen) * width ** -0.5).to(BF).cuda()
    down = (torch.randn(experts, width, inner, generator=gen) * inner ** -0.5).to(BF).cuda()
    ids = torch.stack([torch.randperm(experts, generator=gen)[:top] for _ in range(tokens)]).int().cuda()
    weights = torch.rand(tokens, top, generator=gen).cuda()
    got = ops.moe_experts(h, ids, weights, up, down, limit=7.0, expert=expert, tile_rows=8).double()
    want = plain(h, ids, weights, up, down, expert, 7.0, inner, False)
    # (the result is rounded to 8 bits, a mean of 2^-10 of it, and so is what falls on the other side of a rounding before)
    assert float((got - want).norm() / want.norm()) < 2.0 ** -8


def test_more_tiles_of_few_rows_than_a_grids_dimension_counts():
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(8)
    tokens, top, experts, size = 131100, 4, 5, 16
    h = torch.randn(tokens, size, generator=gen).to(BF).cuda()
    up, down = (torch.randn(experts, size, size, generator=gen).to(BF).cuda() for _ in range(2))
    ids = torch.stack([(torch.arange(tokens) + i) % experts for i in range(top)], dim=1).int().cuda()
    weights = torch.rand(tokens, top, generator=gen).cuda()
    got, want = (ops.moe_experts(h, ids, weights, up, down, expert="relu2", tile_rows=rows).double() for rows in (8, 32))
    assert float((got - want).norm() / want.norm()) < 2.0 ** -8
    for part in (slice(0, 1000), slice(-1000, None)):
        assert float((got[part] - want[part]).norm() / want[part].norm()) < 2.0 ** -8


# by a cluster: its smallest steps, all its experts, the last pairs that its threads keep and the first that they walk twice
@pytest.mark.parametrize("pairs,experts", [(512, 64), (513, 1), (513, 64), (2049, 33), (2049, 65), (16383, 16), (16384, 64), (16385, 16), (40000, 63)])
def test_pairs_are_dealt_to_tiles_by_eight_blocks(pairs, experts):
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(pairs)
    ids = torch.randint(0, experts + 1, (pairs,), generator=gen, dtype=torch.int32)       # (`experts`: an identity expert)
    bm = 16
    tiles = -(-pairs // bm) + min(experts, pairs)
    placed = torch.full((tiles * bm,), -7, dtype=torch.int32, device="cuda")
    tile_expert = torch.full((tiles,), -7, dtype=torch.int32, device="cuda")
    used = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops._check(ops._lib("moe").sb_moe_align(ids.cuda(), pairs, experts, placed, tiles * bm, tile_expert, used, bm, ops._stream()), "moe_align")
    placed, names, used = placed.cpu().view(tiles, bm), tile_expert.cpu(), int(used)
    counts = torch.bincount(ids, minlength=experts + 1)[:experts]
    assert used == int(((counts + bm - 1) // bm).sum())
    assert names[:used].tolist() == sorted(names[:used].tolist())
    for expert in range(experts):
        mine = placed[:used][names[:used] == expert].flatten()
        n = int(counts[expert])
        assert sorted(mine[:n].tolist()) == (ids == expert).nonzero().flatten().tolist()
        assert (mine[n:] == -1).all()
