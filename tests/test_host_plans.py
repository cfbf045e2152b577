"""Host-side planning that needs no device: the step's packed arrays and tile list, the product's
tile/split/stage plan, the decode attention's split count (no GPU)."""

import numpy as np
import pytest

from starter_b200.engine.batch import StepEntry, plan_step


def test_plan_step_packs_sequences_and_lists_query_tiles():
    entries = [StepEntry(3, [5, 6, 7], [0, 2]), StepEntry(0, list(range(130)), [129]), StepEntry(7, [9], [])]
    arrays = plan_step(entries, starts=[10, 0, 64], vocab_size=200)
    assert arrays["tokens"].tolist() == [5, 6, 7] + list(range(130)) + [9]
    assert arrays["tok_pos"].tolist() == [10, 11, 12] + list(range(130)) + [64]
    assert arrays["tok_slot"].tolist() == [3] * 3 + [0] * 130 + [7]
    assert arrays["seq_q_start"].tolist() == [0, 3, 133] and arrays["seq_q_len"].tolist() == [3, 130, 1]
    assert arrays["seq_kv_len"].tolist() == [13, 130, 65]
    assert arrays["want_rows"].tolist() == [0, 2, 3 + 129]
    tiles = list(zip(arrays["tile_seq"].tolist(), arrays["tile_first"].tolist()))
    assert sorted(tiles) == [(0, 0), (1, 0), (1, 64), (1, 128), (2, 0)]
    # the tiles with most keys to walk come first
    keys = [arrays["seq_kv_len"][s] - arrays["seq_q_len"][s] + f for s, f in tiles]
    assert keys == sorted(keys, reverse=True)
    assert all(a.dtype == np.int32 for a in arrays.values())
    # the same list in blocks of 256 queries (what the tensor-core prompt attention launches)
    more = plan_step([StepEntry(0, list(range(600)), []), StepEntry(1, list(range(100)), [])], [0, 300], 1000)
    blocks = list(zip(more["block_seq"].tolist(), more["block_first"].tolist()))
    assert blocks == [(0, 512), (1, 0), (0, 256), (0, 0)]      # most keys first: 512, 300, 256, 0 before them


@pytest.mark.parametrize("entries,starts,message", [
    ([], [], "at least one"),
    ([StepEntry(1, [1], []), StepEntry(1, [2], [])], [0, 1], "twice"),
    ([StepEntry(1, [], [])], [0], "no token"),
    ([StepEntry(1, [1, 2], [2])], [0], "place 2"),
    ([StepEntry(1, [300], [])], [0], "outside the vocabulary"),
])
def test_plan_step_refuses_what_makes_no_sense(entries, starts, message):
    with pytest.raises(ValueError, match=message):
        plan_step(entries, starts, vocab_size=200)


def test_product_plan_keeps_every_cta_resident_and_the_tile_in_the_ring():
    from starter_b200.ops import gemm_plan

    shapes = [(6144, 2560, False), (2560, 4096, False), (9728, 2560, True), (2560, 9728, False),
              (151936, 2560, False), (300, 72, False), (64, 8, True)]
    for rows in (1, 8, 16, 17, 33, 64, 65, 200, 256):
        for n, k, gated in shapes:
            bm, splits, stages = gemm_plan(rows, n, k, gated)
            assert bm in (16, 32, 64, 128) and bm >= min(rows, 128)     # more rows: several row tiles
            assert 1 <= splits <= 8 and 2 <= stages <= 8
            stage_bytes = 16384 + bm * 128
            assert stages * stage_bytes + 1024 <= 227 * 1024
            tiles = (n // 64 if gated else -(-n // 128)) * -(-rows // bm)
            if rows <= 64 and splits > 1:
                per_sm = (227 * 1024) // (stages * stage_bytes + 2048)
                assert tiles * splits <= 148 * per_sm          # one wave


def test_decode_attention_splits_fit_one_wave_and_respect_the_length():
    from starter_b200.ops import decode_splits

    assert decode_splits(1, 8, 4, 16) == 8                       # never more parts than a cluster merges
    assert decode_splits(1, 8, 4, 16, kv_hint=3073) == 8
    assert decode_splits(2, 8, 4, 16, kv_hint=3073) == 8
    assert decode_splits(4, 8, 4, 16, kv_hint=3073) == 7         # 224 blocks rather than 256
    assert decode_splits(5, 8, 4, 16, kv_hint=3073) == 6         # 240 blocks, not 280
    assert decode_splits(6, 8, 4, 16, kv_hint=3073) == 5
    assert decode_splits(8, 8, 4, 16, kv_hint=3073) == 4
    assert decode_splits(12, 8, 4, 16, kv_hint=3073) == 2        # 192 blocks, not 288
    assert decode_splits(1, 8, 4, 16, kv_hint=513) == 8
    assert decode_splits(1, 8, 4, 16, kv_hint=16384) == 32       # one long row: many parts through scratch
    assert decode_splits(1, 8, 4, 16, kv_hint=6000) == 8
    assert decode_splits(2, 8, 4, 16, kv_hint=16384) == 8        # two rows fill the SMs from a cluster
    assert decode_splits(8, 8, 4, 16, kv_hint=130) == 3          # a part is a page at least
    assert decode_splits(64, 8, 4, 16) == 1
    assert decode_splits(1, 8, 4, 16, kv_hint=10) == 1
    assert decode_splits(1, 8, 4, 4, kv_hint=513) == 3           # CUDA-core kernel: three pages a part
    for rows in (1, 2, 3, 5, 7, 8, 9, 10, 30, 64):
        for keys in (0, 700, 3073, 20000):
            assert rows * 8 * decode_splits(rows, 8, 4, 16, kv_hint=keys) <= max(256, rows * 8)


def test_decode_graph_length_classes_never_exceed_the_length():
    """A graph captured for a class assumes the class's shortest length: the class of a length is the
    largest one not above it, so every part of the attention keeps a page or more."""
    from starter_b200.engine.graphs import HINT_PAGES, hint_pages

    assert HINT_PAGES[:8] == (1, 2, 3, 4, 6, 8, 12, 16)
    for tokens in (0, 1, 64, 65, 128, 129, 200, 3073, 4096, 100_000):
        pages = max(1, -(-tokens // 64))
        got = hint_pages(tokens)
        assert got in HINT_PAGES and got <= pages
        assert all(p > pages for p in HINT_PAGES if p > got)
    assert [hint_pages(t) for t in (1, 65, 130, 3073)] == [1, 2, 3, 48]


def test_every_entry_point_the_operations_call_has_declared_arguments():
    """Addresses travel as plain integers: an entry point whose arguments are not declared would cut them to 32 bits."""
    import ctypes
    import inspect
    import re

    from starter_b200 import ops
    from starter_b200.csrc import build

    known = {}
    for name in build.SOURCES:
        known.update(build.declarations(name))
    used = set(re.findall(r"\.(sb_\w+)", inspect.getsource(ops))) - {"sb_page_tokens"}
    assert used and not used - set(known)
    result, types = known["sb_sgemm_nt"]
    assert result is ctypes.c_int
    assert types == [ctypes.c_void_p] * 3 + [ctypes.c_int] * 3 + [ctypes.c_void_p] * 2


@pytest.mark.parametrize("heads, past, new, window, takes", [
    (16, 65000, 64, None, True), (128, 0, 10000, None, True), (128, 0, 30000, None, True), (128, 20000, 64, None, False),
    (128, 9000, 64, None, True), (128, 65000, 64, 4096, True), (128, 65000, 15000, None, False), (128, 65000, 20000, None, False),
    (16, 65537, 64, None, False)])
def test_formed_keys_are_bounded_in_bytes(heads, past, new, window, takes):
    """Beyond the fixed bound they take no more than what the kernel that scores the latents would need."""
    from types import SimpleNamespace

    import torch

    from starter_b200 import ops

    ctx = SimpleNamespace(host={"seq_q_len": np.array([new]), "seq_kv_len": np.array([past + new])}, block_seq=torch.zeros(1))
    got = ops.latent_prompt_takes(torch.bfloat16, ctx, 128, 64, 128, 512, 0.1, window, heads)
    assert got is takes
    if got:
        rows = min(past + new, new + (window or past) - 1) + 64
        assert 2 * rows * (heads * 256 + 576) <= max(ops.LATENT_PROMPT_BYTES, 2 * new * heads * 1088) + 64 * 2 * (heads * 256 + 576)


@pytest.mark.parametrize("heads, news, takes", [
    (16, [32], True), (16, [32] * 8, True), (16, [32] * 16, False), (16, [36] * 16, False), (16, [38] * 16, True), (16, [48] * 32, True),
    (32, [32] * 4, True), (32, [32] * 8, False), (32, [48] * 32, True), (16, [2000] + [32] * 15, True), (16, [31] * 2, False)])
def test_keys_are_formed_where_that_is_the_shorter_way(heads, news, takes):
    """Many sequences of few tokens fill the chip with blocks that score the latents; one block more is a second wave."""
    from types import SimpleNamespace

    import torch

    from starter_b200 import ops

    new = np.array(news, dtype=np.int32)
    for past in (0, 1000):
        ctx = SimpleNamespace(host={"seq_q_len": new, "seq_kv_len": new + past}, block_seq=torch.zeros(1))
        assert ops.latent_prompt_takes(torch.bfloat16, ctx, 128, 64, 128, 512, 0.1, None, heads) is takes


def test_native_entry_points_take_their_declared_arguments():
    """Entries called natively (csrc/host.cpp) hand over what ctypes does: more arguments than registers, 64-bit results, numbers that
    ctypes wraps; anything else is refused before the call."""
    import ctypes

    import torch

    from starter_b200 import ops
    from starter_b200.csrc import build

    native, plain = ops._lib("state_scan_prompt"), build.load("state_scan_prompt")
    assert native.sb_scan_segment_floats(40000, 64) == plain.sb_scan_segment_floats(40000, 64) > 2 ** 28
    for args in ((1, 0, 160, 128, None, 128, 320, 64, 0, 4, 2, 128, 64), (1, 1, 160, 128, 0, 128, 320, 64, None, 4, 2, 120, 64),
                 (1, 2, 160, 128, 0, 128, 328, 64, None, 4, 4, 128, 64), (0, 2, 160, 128, 0, 128, 328, 64, None, 4, 4, 128, 64)):
        assert native.sb_scan_prompt_floats(*args) == plain.sb_scan_prompt_floats(*args)
    assert native.sb_scan_segment_floats(ctypes.c_int(3), 64) == plain.sb_scan_segment_floats(3, 64)
    x = torch.zeros(4)
    assert native.sb_scan_prompt_floats(1, 0, x, 128, x, 128, x, 64, None, 4, 2, 128, 64) == 4 * 20
    with pytest.raises(TypeError):
        native.sb_scan_segment_floats(3)
    for bad in (x, 1.5, "3", None):
        with pytest.raises(TypeError):
            native.sb_scan_segment_floats(3, bad)


def test_native_entry_points_take_what_stands_for_a_number():
    """Sizes and factors that come as numpy's numbers, tensors of one, or objects with ``__index__``, as ctypes takes them."""
    import ctypes

    import torch

    from starter_b200 import ops
    from starter_b200.csrc import build

    class Four:
        def __index__(self):
            return 4

    native, plain = ops._lib("state_scan_prompt"), build.load("state_scan_prompt")
    for four in (np.int64(4), np.int32(4), np.uint8(4), np.array(4), torch.tensor(4), torch.tensor([4]), Four(), True):
        assert native.sb_scan_segment_floats(four, 64) == plain.sb_scan_segment_floats(four, 64)
    for bad in (np.float32(4), torch.tensor(4.0), torch.tensor([1, 2]), 4.0):
        with pytest.raises((TypeError, ctypes.ArgumentError)):
            plain.sb_scan_segment_floats(bad, 64)
        with pytest.raises(TypeError):
            native.sb_scan_segment_floats(bad, 64)
    # (no rows: the entry point returns before it looks further)
    for eps in (np.float32(1e-6), np.float64(1e-6), torch.tensor(1e-6), 0, ctypes.c_float(1e-6)):
        assert ops._lib("elementwise").sb_rmsnorm(0, 0, None, None, None, None, None, 0, 64, eps, None) == 0
    for bad in (None, "1e-6", torch.zeros(2)):
        with pytest.raises(TypeError):
            ops._lib("elementwise").sb_rmsnorm(0, 0, None, None, None, None, None, 0, 64, bad, None)


def test_native_checks_refuse_what_the_plain_ones_do():
    import torch

    from starter_b200 import ops

    ops._bind()
    for bad in (torch.zeros(2, 2), None, 3, [1.0]):
        with pytest.raises(ops.KernelError, match="x must be a CUDA tensor"):
            ops._need(bad, "x", torch.float32, 2)
    assert ops._empty(torch.zeros(2), (3, 5), torch.int32).shape == (3, 5)
    assert ops._empty(torch.zeros(2, dtype=torch.bfloat16), (0, 5)).dtype == torch.bfloat16
    with pytest.raises((RuntimeError, TypeError)):
        ops._empty(torch.zeros(2), (-3, 5))


def test_warps_are_whole_in_front_of_aligned_cluster_barriers():
    """``barrier.cluster`` with ``.aligned`` wants all threads of a warp at it at once: in every kernel source the statement in front of
    one makes the warp whole (a loop that lanes leave at different rounds need not)."""
    import os
    import re

    from starter_b200.csrc import build

    barriers = 0
    for name in sorted(os.listdir(build.HERE)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(build.HERE, name)) as handle:
            code = [re.sub(r"\s*//.*", "", line).strip() for line in handle]
        code = [line for line in code if line]
        for i, line in enumerate(code):
            if "barrier.cluster." in line and ".aligned" in line:
                barriers += 1
                assert re.search(r"__sync(warp|threads)\(\);$", code[i - 1]), f"{name}: {code[i - 1]!r} in front of {line!r}"
    assert barriers >= 4


def test_steps_whose_latent_products_are_for_few_rows():
    """Both head-wise kernels up to 8 single tokens and 64 of prompts, the queries' alone up to 16 single tokens."""
    import torch

    from starter_b200 import ops

    for n, longest, takes in ((1, 1, (True, True)), (8, 1, (True, True)), (9, 1, (True, False)), (16, 1, (True, False)), (17, 1, (False, False)),
                              (64, 1, (False, False)), (9, 2, (True, True)), (64, 33, (True, True)), (65, 33, (False, False))):
        assert ops.latent_heads_take(torch.empty(n, 8, dtype=torch.bfloat16), 128, 64, 512, 128, longest) == takes
        assert ops.latent_heads_take(torch.empty(n, 8), 128, 64, 512, 128, longest) == (False, False)
        assert ops.latent_heads_take(torch.empty(n, 8, dtype=torch.bfloat16), 120, 64, 512, 128, longest) == (False, False)


@pytest.mark.parametrize("up", [0, 1, 2])
def test_products_over_tiles_of_eight_rows_come_in_pairs(up):
    """The down product of few rows reads its tiles in front of its wait, so neither of the two has an entry of its own."""
    from starter_b200.csrc import build

    entry = build.load("moe").sb_moe_tiles
    result, types = build.declarations("moe")["sb_moe_tiles"]
    entry.restype, entry.argtypes = result, types
    tile_rows = 8
    # (refused in front of any launch, so no address is looked at)
    assert entry(1, up, tile_rows, None, None, None, None, None, None, 1, 64, 64, 1, 0.0, None, None) == -2


def test_the_router_takes_sixteen_tokens_a_block_behind_a_wave_of_four_a_block():
    from starter_b200.csrc import build

    entry = build.load("moe").sb_moe_route_many_from
    # (two blocks of four an SM with more than 16 experts: 1,184 tokens of 64 experts 16 us, in sixteens 27)
    assert [entry(n) for n in (1, 16, 17, 64)] == [592, 592, 1185, 1185]


def test_queries_are_turned_beside_the_gathering_where_its_grid_holds_them():
    from starter_b200.csrc import build
    from starter_b200.ops import latent_turn_rows

    assert latent_turn_rows(2048, 16, 1, 2048) == 1 + 4 and latent_turn_rows(33, 3, 2, 64) == 2 + 1
    # (252 heads and 1,024 sequences of 64 tokens, which the path takes: a row too many for one grid)
    assert latent_turn_rows(65536, 251, 1024, 64) <= 65535 < latent_turn_rows(65536, 252, 1024, 64)
    entry = build.load("attention_latent_prompt").sb_latent_gather
    result, types = build.declarations("attention_latent_prompt")["sb_latent_gather"]
    entry.restype, entry.argtypes = result, types
    at = 4096              # (no address is looked at: the entry refuses in front of its launch)
    assert entry(at, at, 1, at, at, at, 1024, 64, at, at, 64, 64, 0, at, at, at, 32, at, 65536, 252, 128, None) == -2
