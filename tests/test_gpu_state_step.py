"""One token a sequence of the matrix-state recurrences with their decays and norms in one kernel, against 64 bits: rows and columns
where a warp's rows, its parts and the block's warps change, shared query/key heads, sequences that bring nothing, and operands off their
alignment, which take the separate kernels."""

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
HALF_STEP = 2.0 ** -8 * 1.01     # rounding to bfloat16 and a little for the sums in 32 bits
F = torch.float64


def step(mode, x, cols, w, S, heads, groups, N, V, gate, gain, parts, gate_first):
    """``(normed rows, their sizes, states)`` in 64 bits of rows ``x`` and states ``S`` ``[n, heads, N, V]``."""
    n, x = x.shape[0], x.to(F)
    q = x[:, cols["q"]:cols["q"] + groups * N].view(n, groups, N).repeat_interleave(heads // groups, dim=1)
    k = x[:, cols["k"]:cols["k"] + groups * N].view(n, groups, N).repeat_interleave(heads // groups, dim=1)
    v = x[:, cols["v"]:cols["v"] + heads * V].view(n, heads, V)
    w = {name: t.to(F) for name, t in w.items()}
    if mode in ("state_space", "gated_delta"):
        dt = torch.logaddexp(x[:, cols["a"]:cols["a"] + heads] + w["dt_bias"], torch.zeros(1, dtype=F, device="cuda"))
        S = S * torch.exp(-torch.exp(w["A_log"]) * dt)[..., None, None]
        if mode == "state_space":
            write = dt[..., None] * v
        else:
            q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * N ** -0.5
            k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
            write = torch.sigmoid(x[:, cols["b"]:cols["b"] + heads])[..., None] * (v - (k[..., None, :] @ S)[..., 0, :])
    elif mode == "forget_write":
        q = q * torch.sigmoid(q)
        f = w["A_log"] + (1 - w["A_log"]) * torch.sigmoid(k.flatten(1) + w["dt_bias"])
        S, k, write = S * f.view(n, heads, N, 1), 1 - f.view(n, heads, N), v
    else:
        z = x[:, cols["low"]:cols["low"] + w["a2"].shape[0]] @ w["a2"] + w["a2_bias"]
        S = S * torch.exp(torch.nn.functional.logsigmoid(z) / 16).view(n, heads, N, 1)
        q, write = q * N ** -0.5, v
    S = S + k[..., None] * write[..., None, :]
    terms = q[..., None] * S
    o, size = terms.sum(-2), terms.abs().sum(-2)
    if mode == "state_space":
        o = o + w["D"][:, None] * v
    g = torch.nn.functional.silu(x[:, cols["g"]:cols["g"] + heads * V]) if gate else torch.ones_like(o.flatten(1))
    y = o.flatten(1) * g if gate_first else o.flatten(1)
    y = y.view(n, parts, -1)
    inv = 1 / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-6)
    gains = w["gain"].repeat(heads * V // w["gain"].shape[0])
    small = (size.flatten(1) * g.abs()).view(n, parts, -1) * inv
    return (y * inv).flatten(1) * gains * (1 if gate_first else g), small.flatten(1) * gains.abs(), S


@pytest.mark.parametrize("heads, groups, N, V", [(4, 4, 128, 128), (4, 2, 72, 128), (3, 3, 8, 128), (4, 1, 128, 64), (2, 2, 16, 64),
                                                 (4, 4, 128, 32), (2, 1, 96, 32)])
@pytest.mark.parametrize("mode", ["state_space", "gated_delta", "forget_write", "channel_decay"])
@pytest.mark.parametrize("aligned", [True, False])
def test_one_token_steps(mode, heads, groups, N, V, aligned):
    from starter_b200 import ops

    if mode in ("forget_write", "channel_decay"):
        groups = heads
    gen = torch.Generator().manual_seed(N + V)
    rank, cols, at = 5 if V == 64 else 37, {}, 0 if aligned else 1
    for name, width in (("q", groups * N), ("k", groups * N), ("v", heads * V), ("g", heads * V), ("a", heads), ("b", heads), ("low", rank)):
        cols[name], at = at, at + width
    rand = lambda *shape: torch.randn(*shape, generator=gen).cuda()
    slots, starts, lens = [4, 0, 2, 1], [0, 1, 2, 2], [1, 1, 0, 1]          # the third brings nothing
    x = rand(3, -(-at // 8) * 8).to(BF)
    w = {"A_log": rand(heads), "dt_bias": rand(heads), "D": rand(heads), "a2": rand(rank, heads * N), "a2_bias": rand(heads * N) + 2}
    if mode == "forget_write":
        w["A_log"], w["dt_bias"] = torch.rand(heads * N, generator=gen).cuda() * 0.5, rand(heads * N)
    gate, gate_first = mode != "forget_write", mode == "state_space"
    parts = 1 if mode == "state_space" else heads
    w["gain"] = rand(heads * V if mode == "state_space" else V)
    state = rand(5, 4 + heads * N * V)
    before = state.clone()
    ints = lambda t: torch.tensor(t, dtype=torch.int32, device="cuda")
    two = mode in ("state_space", "gated_delta")
    counted = ops.launch_count
    got = ops.state_scan_norm(mode, (x, cols["q"]), (x, cols["k"]), (x, cols["v"]), (x, cols["a"]) if two else None,
                              (x, cols["b"]) if mode == "gated_delta" else None, w["A_log"] if mode != "channel_decay" else None,
                              w["dt_bias"] if mode != "channel_decay" else None, w["D"] if mode == "state_space" else None, state, 4,
                              ints(slots), ints(starts), ints(lens), 1, heads, groups, N, V, w["gain"], parts, 1e-6,
                              gate=(x, cols["g"]) if gate else None, gate_first=gate_first,
                              low=(x, cols["low"], w["a2"], w["a2_bias"], 16.0) if mode == "channel_decay" else None)
    launched = ops.launch_count - counted
    assert launched == (1 if aligned else 2 + (mode == "channel_decay")) + (aligned and mode == "state_space")
    here = [4, 0, 1]
    S = before[here, 4:].view(3, heads, N, V).to(F)
    want, size, S = step(mode, x, cols, w, S, heads, groups, N, V, gate, None, parts, gate_first)
    # (the sums' terms in 32 bits, and where a decay is formed: exponentials of sums of up to 40)
    assert bool(((got.to(F) - want).abs() <= HALF_STEP * want.abs() + 2.0 ** -17 * size).all())
    left = state[here, 4:].view(3, heads, N, V).to(F)
    bound = 2.0 ** -18 * (S.abs() + before[here, 4:].view(3, heads, N, V).to(F).abs() + S.abs().amax(-2, keepdim=True))
    assert bool(((left - S).abs() <= bound).all())
    assert torch.equal(state[[2, 3]], before[[2, 3]]) and torch.equal(state[:, :4], before[:, :4])


@pytest.mark.parametrize("dtype", [BF, torch.float32])
def test_low_rank_entries_of_either_type(dtype):
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(5)
    n, heads, N, V, rank = 3, 2, 64, 64, 12
    rand = lambda *shape: torch.randn(*shape, generator=gen).cuda()
    x, low, a2, bias, gain = rand(n, 4 * heads * N).to(BF), rand(n, rank).to(dtype), rand(rank, heads * N), rand(heads * N) + 2, rand(V)
    ints = lambda t: torch.tensor(t, dtype=torch.int32, device="cuda")
    at, w = heads * N, {"a2": a2, "a2_bias": bias, "gain": gain}
    state = rand(n, heads * N * V)
    before = state.clone().view(n, heads, N, V).to(F)
    got = ops.state_scan_norm("channel_decay", (x, 0), (x, at), (x, 2 * at), None, None, None, None, None, state, 0, ints([0, 1, 2]),
                              ints([0, 1, 2]), ints([1, 1, 1]), 1, heads, heads, N, V, gain, heads, 1e-6, gate=(x, 3 * at),
                              low=(low, 0, a2, bias, 16.0))
    cols = {"q": 0, "k": at, "v": 2 * at, "g": 3 * at, "low": 4 * at}
    want, size, S = step("channel_decay", torch.cat([x.to(F), low.to(F)], dim=1), cols, w, before, heads, heads, N, V, True, gain, heads, False)
    assert bool(((got.to(F) - want).abs() <= HALF_STEP * want.abs() + 2.0 ** -17 * size).all())
    left = state.view(n, heads, N, V).to(F)
    assert bool(((left - S).abs() <= 2.0 ** -18 * (S.abs() + before.abs() + S.abs().amax(-2, keepdim=True))).all())
