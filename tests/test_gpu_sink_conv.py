"""The window attention's convolution, norms, rotation and cache write in one kernel against the two kernels that it stands for: both numbers
of tokens a thread, warps of queries, keys and values of several sizes, one to four taps, sequences of few and many tokens."""

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("heads, kv, dim, vdim, rot, width", [(2, 1, 128, 128, 128, 0), (4, 2, 64, 64, 32, 8), (16, 8, 128, 128, 128, 0),
                                                              (16, 4, 128, 128, 0, 0), (4, 2, 128, 64, 8, 0), (3, 1, 64, 64, 64, 0)])
@pytest.mark.parametrize("taps", [1, 2, 3, 4])
@pytest.mark.parametrize("norm, bias", [(True, True), (True, False), (False, True)])
@pytest.mark.parametrize("sizes", [[1, 3, 2, 9], [600, 601]])
def test_one_kernel_gives_what_two_give(heads, kv, dim, vdim, rot, width, taps, norm, bias, sizes):
    from starter_b200 import ops
    from starter_b200.config import InterleavedRopeSpec
    from starter_b200.parts import InterleavedRotaryTable

    gen = torch.Generator().manual_seed(heads + 7 * taps + sizes[0])
    rand = lambda *shape: torch.randn(*shape, generator=gen).cuda()
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    channels, n, past = heads * dim + kv * (dim + vdim), len(sizes), 5
    proj = rand(sum(sizes), channels + width).to(BF)
    w, in_bias = rand(channels, taps), rand(channels) if bias else None
    gains = (rand(heads * dim), rand(kv * dim)) if norm else None
    tables = InterleavedRotaryTable(InterleavedRopeSpec(dims=rot, base=100.0), BF, "cuda") if rot else None
    if rot:
        tables.ensure(700)
    state = rand(n + 1, 4 + (taps - 1) * channels) if taps > 1 else None
    slots, starts = list(range(n, 0, -1)), [sum(sizes[:i]) for i in range(n)]
    pos = ints([past + t for s in sizes for t in range(s)])
    slot = ints([slots[i] for i, s in enumerate(sizes) for _ in range(s)])
    per = -(-(max(sizes) + past) // 64)
    table = torch.randperm((n + 1) * per, generator=gen).int().view(n + 1, per).cuda()
    stores = [torch.zeros((n + 1) * per, kv, 64, d, dtype=BF, device="cuda") for d in (dim, vdim)]
    other, kept = [t.clone() for t in stores], state.clone() if taps > 1 else None
    seqs = (ints(slots), ints(starts), ints(sizes), max(sizes))
    rotation = tables.rotation() if rot else None
    counted = ops.launch_count
    q = ops.sink_conv_prepare(proj, w, in_bias, state, 4 if taps > 1 else 0, *seqs, heads, kv, dim, vdim, pos, slot, table, *stores, rotation, gains,
                              eps=1e-6)
    assert ops.launch_count - counted == (1 if heads != 3 else 2)
    want = ops.short_conv(proj, 0, channels, w, None, in_bias, kept, 4 if taps > 1 else 0, *seqs)
    ops.sink_prepare_norm(want, heads, kv, dim, vdim, pos, slot, table, *other, rotation, gains, False, 1e-6)
    # the convolved values are the same bits; the rows' sums of squares meet in another order, which may move a rounding to 8 bits
    for got, ref in ((q[:, :heads * dim], want[:, :heads * dim]), (stores[0], other[0])):
        got, ref = got.double(), ref.double()
        assert bool(((got - ref).abs() <= 2.0 ** -7 * ref.abs() + 2.0 ** -22 * ref.abs().amax(-1, keepdim=True)).all())
        assert float((got != ref).double().mean()) < 1e-3
    assert torch.equal(stores[1], other[1])
    assert state is None or torch.equal(state, kept)


@pytest.mark.parametrize("which", ["tok_pos", "tok_slot"])
def test_places_of_another_type_are_refused(which):
    from starter_b200 import ops

    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    heads, kv, dim = 2, 1, 128
    channels, places = heads * dim + 2 * kv * dim, {"tok_pos": ints([0, 1]), "tok_slot": ints([0, 0])}
    places[which] = places[which].long()
    stores = [torch.zeros(1, kv, 64, dim, dtype=BF, device="cuda") for _ in range(2)]
    with pytest.raises(ops.KernelError, match=which):
        ops.sink_conv_prepare(torch.zeros(2, channels, dtype=BF, device="cuda"), torch.zeros(channels, 1, device="cuda"), None, None, 0, ints([0]),
                              ints([0]), ints([2]), 2, heads, kv, dim, dim, places["tok_pos"], places["tok_slot"], ints([[0]]), *stores, eps=1e-6)
