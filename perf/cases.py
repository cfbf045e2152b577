"""What this library's speed is measured on: the work its users have it do, case by case.

Most cases are one layer part (a mixer, a feed-forward) called as a program that composes parts calls it: the
part, its weights, a sequence cache and a step's context are what such a program keeps; the call is the part's.
A step of one token per sequence is captured in a CUDA graph first, as the engine captures its own, because that is
how such steps are run.  Two kinds of case are whole calls: ``ModelRunner.step`` on unequal prompts and
``ModelRunner.decode_tokens`` on a batch of running sequences, with the logits they leave.

Sizes are those of the design comparisons of ``bench.py`` (width 2048, 16 heads of 128 on 4 key/value heads, a latent of
512, states of 128, 16 experts of which a token uses 4) and of its headline model (width 2560, 32 heads on 8, a
feed-forward of 9,728); the whole calls run four of its layers under the full vocabulary.
"""

import math

import torch

from starter_b200 import ops  # noqa: F401  (the kernels: a missing library shows here, not in a timed pass)
from starter_b200.cache import SequenceCache
from starter_b200.config import config_from_dict
from starter_b200.config import spec as S
from starter_b200.engine import ModelRunner, StepContext, StepEntry, plan_step, random_model
from starter_b200.engine.batch import upload
from starter_b200.parts import lookup
from starter_b200.weights import random_checkpoint, random_tensor

DEVICE = "cuda:0"
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
RECURRENT = ("state_space", "gated_delta", "forget_write", "gated_linear_attention")


# ------------------------------------------------------------------------------------------ the cases

def listed():
    model = dict(kind="model", dtype="bf16", layers=4, width=2560, heads=32, kv_heads=8, ff=9728, vocab=151936)
    design = dict(dtype="bf16", width=2048, heads=16, kv_heads=4)
    return [
        # the decoding of a small batch, far into unequal sequences: what generation spends its time on
        dict(model, name="model_decode", seqs=8, new=1, past=3072, ragged=True),
        # a few unequal prompts in one step, as a batch of requests starts
        dict(model, name="model_prompts", seqs=3, new=900, past=0, ragged=True),
        # a later portion of a long prompt, of a few hundred tokens: attention over what is cached, then the feed-forward
        dict(design, kind="dense", name="dense_portion", seqs=1, new=300, past=1000, ragged=False, ff=8192),
        # the 32-bit path, for which short prompts and trace replays are run
        dict(design, kind="dense", name="dense_float32", dtype="fp32", seqs=2, new=77, past=0, ragged=True, ff=4096),
        # attention over a cached latent: a prompt, and single tokens of a running batch
        dict(design, kind="latent", name="latent_prompt", seqs=1, new=2048, past=0, ragged=False, rank=512, window=0, sink=True),
        dict(design, kind="latent", name="latent_decode", seqs=8, new=1, past=2048, ragged=True, rank=512, window=0, sink=True),
        # window attention with biases, short convolutions, row norms, capped scores and a sink: a prompt
        dict(design, kind="window", name="window_prompt", seqs=1, new=2048, past=0, ragged=False, window=1024, cap=50.0, sink=True),
        # recurrences with a matrix state per head: prompts (one long one, unequal ones), a single token of one sequence
        dict(design, kind="state_space", name="state_space_prompt", seqs=1, new=2048, past=0, ragged=False),
        dict(design, kind="gated_delta", name="delta_prompts", seqs=3, new=801, past=0, ragged=True),
        dict(design, kind="gated_linear_attention", name="linear_attention_step", seqs=1, new=1, past=100, ragged=False),
        # routed experts: a prompt's tokens, and those of a running batch
        dict(design, kind="experts", name="experts_prompt", seqs=1, new=2048, past=0, ragged=False, ff=2048, experts=16, top=4,
             expert="gated_silu"),
        dict(design, kind="experts", name="experts_decode", seqs=8, new=1, past=0, ragged=False, ff=2048, experts=16, top=4,
             expert="gated_silu"),
    ]


def _spread(rng, low, high):
    """A whole number from ``low`` to ``high``, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("model", "dense", "dense", "latent", "latent", "window", "window", "recurrent", "recurrent", "recurrent",
                       "experts", "experts"))
    if kind == "model":
        case = dict(kind="model", dtype="bf16", layers=rng.randint(1, 4), width=2560, heads=32, kv_heads=8,
                    ff=64 * rng.randint(64, 152), vocab=rng.choice((32768, 151936)))
        if rng.random() < 0.5:
            return dict(case, seqs=_spread(rng, 1, 16), new=1, past=_spread(rng, 50, 1500), ragged=True)
        seqs = rng.randint(1, 4)
        return dict(case, seqs=seqs, new=_spread(rng, 60, 2000 // seqs), past=0, ragged=True)
    if kind == "recurrent":
        kind = rng.choice(RECURRENT)
    case = dict(kind=kind, dtype="fp32" if kind == "dense" and rng.random() < 0.3 else "bf16", width=128 * rng.randint(8, 16),
                heads=16, kv_heads=rng.choice((4, 8)))
    if kind in RECURRENT:
        case["heads"] = rng.choice((8, 12, 16))
    if rng.random() < 0.4:      # single tokens of a running batch
        case.update(seqs=_spread(rng, 1, 32), new=1, past=_spread(rng, 40, 1500))
    elif rng.random() < 0.3:    # a later portion
        case.update(seqs=rng.randint(1, 2), new=_spread(rng, 17, 700), past=_spread(rng, 40, 1200))
    else:                       # prompts
        seqs = rng.randint(1, 4)
        case.update(seqs=seqs, new=_spread(rng, 40, 2000 // seqs), past=0)
    case["ragged"] = rng.random() < 0.7
    if case["dtype"] == "fp32":
        case.update(new=min(case["new"], 150), past=min(case["past"], 150), seqs=min(case["seqs"], 2))
    if kind == "dense":
        case["ff"] = 64 * rng.randint(32, 64 if case["dtype"] == "fp32" else 128)
    elif kind == "latent":
        case.update(rank=rng.choice((256, 512)), window=rng.choice((0, 0, 512, 1024)), sink=rng.random() < 0.5)
    elif kind == "window":
        case.update(window=rng.choice((256, 1000, 1024)), cap=rng.choice((0.0, 50.0)), sink=rng.random() < 0.5)
    elif kind == "experts":
        case.update(ff=64 * rng.randint(12, 32), experts=rng.choice((8, 16, 32)), top=rng.randint(2, 4), past=0,
                    expert=rng.choice(("gated_silu", "relu2", "gated_clamped")))
    return case


def _lengths(case):
    """``[(cached tokens, new tokens)]`` of the case's sequences; ragged ones differ by about a third."""
    out = []
    for i in range(case["seqs"]):
        share = 1.0 - (i / (3.0 * case["seqs"]) if case["ragged"] else 0.0)
        past = max(1, int(case["past"] * share) - (i if case["ragged"] else 0)) if case["past"] else 0
        out.append((past, max(1, int(case["new"] * share))))
    return out


def _captured(case):
    """Steps of one token per sequence are captured."""
    return case["new"] == 1


# ------------------------------------------------------------------------------------------ specs, weights, inputs

def _specs(case):
    """``[(family, spec)]`` of the parts a case calls, the mixer first."""
    kind, width, heads = case["kind"], case["width"], case["heads"]
    if kind == "dense":
        return [("mixer", S.AttentionSpec(width, heads, case["kv_heads"], 128, 128 ** -0.5, True, 1e-6, S.RopeSpec(128, 1e6))),
                ("feed_forward", S.GatedFeedForwardSpec(width, case["ff"]))]
    if kind == "latent":
        return [("mixer", S.LatentAttentionSpec(width, heads, 128, 64, 128, width * 3 // 4 // 64 * 64, case["rank"], 192 ** -0.5,
                                                1e-6, S.InterleavedRopeSpec(64, 1e4), window=case["window"] or None,
                                                sink=case["sink"], output_gate=True))]
    if kind == "window":
        return [("mixer", S.SinkAttentionSpec(width, heads, case["kv_heads"], 128, 128, 128 ** -0.5, distance_penalty=False,
                                              sink=case["sink"], head_gate=False, window=case["window"],
                                              position=S.InterleavedRopeSpec(128, 1e6), softcap=case["cap"] or None, bias=True,
                                              conv=3, row_norm=True, norm_eps=1e-6))]
    if kind == "state_space":
        return [("mixer", S.StateSpaceSpec(width, 2 * heads, 64, 128, 1, 4, 1, 1e-6))]
    if kind == "gated_delta":
        return [("mixer", S.GatedDeltaSpec(width, heads, heads // 2, 128, 128, 4, 1e-6))]
    if kind == "forget_write":
        return [("mixer", S.ForgetWriteSpec(width, heads, 128, 128, 1e-6))]
    if kind == "gated_linear_attention":
        return [("mixer", S.GatedLinearAttentionSpec(width, heads, 128, 128, 16.0, 16, 1e-6))]
    if kind == "experts":
        scoring = dict(gated_silu=("sigmoid", 1.0, False), relu2=("sigmoid_normalised", 2.5, False),
                       gated_clamped=("softmax_top", 1.0, True))[case["expert"]]
        return [("feed_forward", S.RoutedExpertsSpec(width, case["ff"], case["experts"], case["top"], limit=7.0,
                                                     expert=case["expert"], scoring=scoring[0], weight_scale=scoring[1],
                                                     router_bias=scoring[2]))]
    raise ValueError(f"no case kind {kind!r}")


def _weights(part, seed, index, dtype):
    """Random weights by their roles: matrices N(0, 0.02), gains around one."""
    out = {}
    for name, p in part.param_specs().items():
        always = p.role in ("gain32", "bias32", "slope", "vector32", "floor", "matrix32")
        out[name] = random_tensor(seed, f"{index}.{name}", p, torch.float32 if always else dtype, DEVICE)
    return out


def _inputs(case, seed):
    """Per sequence the rows in front of the step and those of the step: what a norm hands to a layer."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed * 7919 + 1)
    dtype, rows = DTYPES[case["dtype"]], []
    for past, new in _lengths(case):
        x = torch.randn((past + new, case["width"]), generator=gen, device=DEVICE).to(dtype)
        rows.append((x[:past], x[past:]))
    return rows


def _parts(case, seed):
    dtype, parts, weights = DTYPES[case["dtype"]], [], []
    for index, (family, spec) in enumerate(_specs(case)):
        cls = lookup(family, spec.kind)
        if family == "mixer":
            where = getattr(spec, "position", None)
            part = cls(spec, dtype, lookup("position", where.kind)(where, dtype, DEVICE) if where is not None else None)
        else:
            part = cls(spec, dtype)
        weights.append(_weights(part, seed, index, dtype))
        part.set_params(dict(weights[-1]))
        parts.append(part)
    return parts, weights


def _context(cache, status, entries):
    """A step's context for entries ``(slot, tokens)``."""
    entries = [StepEntry(slot, [0] * n, []) for slot, n in entries]
    arrays = plan_step(entries, [cache.lengths[e.slot] for e in entries])
    for e in entries:
        cache.reserve(e.slot, cache.lengths[e.slot] + len(e.tokens))
        cache.advance(e.slot, len(e.tokens))
    cache.sync_table()
    dev = upload(arrays, torch.device(DEVICE))
    return StepContext(n_tokens=int(arrays["tokens"].size), n_seqs=len(entries), max_q_len=int(arrays["seq_q_len"].max()),
                       max_kv_len=int(arrays["seq_kv_len"].max()), cache=cache, status=status, host=arrays,
                       **{k: dev[k] for k in ("tokens", "tok_pos", "tok_slot", "seq_slot", "seq_q_start", "seq_q_len",
                                              "seq_kv_len", "want_rows", "tile_seq", "tile_first", "block_seq", "block_first")})


def _tokens(case, seed):
    gen = torch.Generator().manual_seed(seed * 7919 + 2)
    return [torch.randint(0, case["vocab"], (past + new,), generator=gen).tolist() for past, new in _lengths(case)]


def _model_config(case):
    return config_from_dict(dict(
        architectures=["Qwen3ForCausalLM"], num_hidden_layers=case["layers"], hidden_size=case["width"],
        num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"], head_dim=128, intermediate_size=case["ff"],
        vocab_size=case["vocab"], rope_theta=5e6, rms_norm_eps=1e-6, tie_word_embeddings=True, max_position_embeddings=4096))


# ------------------------------------------------------------------------------------------ prepare and run

def prepare(case, seed):
    if case["kind"] == "model":
        return _prepare_model(case, seed)
    parts, _ = _parts(case, seed)
    rows, lengths = _inputs(case, seed), _lengths(case)
    heads = case["heads"]
    shape = (2 * heads, 128, 64) if case["kind"] == "state_space" else (heads if case["kind"] in RECURRENT else 0, 128, 128)
    state = {"case": case, "shape": shape, "parts": parts, "x": torch.cat([new for _, new in rows]), "ctx": None, "graph": None}
    mixer = parts[0] if hasattr(parts[0], "kv_need") else None
    if mixer is not None:
        total = sum(-(-(past + new) // 64) * 64 for past, new in lengths)
        cache = SequenceCache({0: mixer.kv_need()}, {0: mixer.state_need()}, total, len(lengths), DTYPES[case["dtype"]], DEVICE)
        status = torch.zeros((1,), dtype=torch.int32, device=DEVICE)
        slots = [cache.open_sequence() for _ in lengths]
        if slots != list(range(len(slots))):
            raise RuntimeError("a new cache hands out its slots in order")
        mixer.prepare(max(past + new for past, new in lengths))
        if case["past"]:
            # what the sequences hold already came through the same layer
            mixer(torch.cat([past for past, _ in rows]), _context(cache, status, [(s, n[0]) for s, n in zip(slots, lengths)]), 0)
        state["ctx"] = _context(cache, status, [(s, n[1]) for s, n in zip(slots, lengths)])
        state["cache"] = cache
    if _captured(case):
        _capture(state)
    return state


def _capture(state):
    """The call as a CUDA graph; what warming it up changes is put back."""
    kept = state["cache"].entry_state(0) if "cache" in state else None
    saved = kept.clone() if kept is not None else None
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side), torch.inference_mode():
        _call(state)
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    if kept is not None:
        kept.copy_(saved)
    graph = torch.cuda.CUDAGraph()
    with torch.inference_mode(), torch.cuda.graph(graph):
        state["out"] = _call(state)
    state["graph"] = graph


def _call(state):
    """The parts' calls and what they leave: outputs, and the cache's keys, values and state."""
    x, ctx, out = state["x"], state["ctx"], {}
    for index, part in enumerate(state["parts"]):
        out[f"y{index}"] = part(x, ctx, 0) if hasattr(part, "kv_need") else part(x, ctx)
    if ctx is not None:
        kept = ctx.cache.entry_state(0)
        if kept is not None:
            # a slot's floats: a convolution's last inputs, then the recurrence's matrices
            shape = state["shape"]
            convolved = kept.shape[1] - math.prod(shape)
            if convolved:
                out["taps"] = kept[:, :convolved]
            if shape[0]:
                out["recurrent"] = kept[:, convolved:].unflatten(1, shape)
        if ctx.cache.groups:
            keys, values = ctx.cache.entry_pages(0)
            out["keys"] = keys
            if values.numel():
                out["values"] = values
    return out


def _prepare_model(case, seed):
    lengths, tokens = _lengths(case), _tokens(case, seed)
    model = random_model(_model_config(case), seed, DTYPES[case["dtype"]], DEVICE)
    total = sum(-(-(past + new) // 64) * 64 for past, new in lengths)
    runner = ModelRunner(model, max_tokens=total, max_sequences=len(lengths))
    state = {"case": case, "runner": runner, "tokens": tokens}
    if _captured(case):
        state["slots"] = [runner.open_sequence() for _ in lengths]
        for slot, seq in zip(state["slots"], tokens):
            runner.step([StepEntry(slot, seq[:-1], [])])
        state["entries"] = [StepEntry(slot, [seq[-1]], [0]) for slot, seq in zip(state["slots"], tokens)]
        _decode(state)      # captures the step
    return state


def _decode(state):
    runner, entries = state["runner"], state["entries"]
    for entry, seq in zip(entries, state["tokens"]):
        runner.cache.lengths[entry.slot] = len(seq) - 1     # the same place of the same sequences in every pass
    drawn = runner.decode_tokens(entries, [0.0] * len(entries), [0] * len(entries))
    return {"logits": runner.graphs.logits[runner.graphs.last_key], "tokens": drawn}


@torch.inference_mode()
def run(state):
    if "runner" not in state:
        if state["graph"] is None:
            return _call(state)
        state["graph"].replay()
        return state["out"]
    if "entries" in state:
        out = _decode(state)
        return {"logits": out["logits"]}
    runner = state["runner"]
    slots = [runner.open_sequence() for _ in state["tokens"]]
    logits = runner.step([StepEntry(slot, seq, [len(seq) - 1]) for slot, seq in zip(slots, state["tokens"])])
    for slot in slots:
        runner.close_sequence(slot)
    return {"logits": logits}


# ------------------------------------------------------------------------------------------ what a pass cannot do without

def _seen(past, new, window=0):
    """Keys seen by the ``new`` queries behind ``past`` tokens, summed; and the distinct keys read."""
    total = sum(min(past + i + 1, window) if window else past + i + 1 for i in range(new))
    return total, min(past + new, window + new) if window else past + new


def work(case):
    lengths, size = _lengths(case), 4 if case["dtype"] == "fp32" else 2
    tokens = sum(new for _, new in lengths)
    width, heads, groups = case["width"], case["heads"], case["kv_heads"]
    kind = case["kind"]
    if kind in ("model", "dense"):
        layer = width * 128 * (2 * heads + 2 * groups)
        ff = 3 * width * case["ff"]
        seen = [_seen(past, new) for past, new in lengths]
        kv_bytes = sum(keys for _, keys in seen) * 2 * groups * 128 * size
        pairs = sum(n for n, _ in seen)
        flops = 2 * tokens * (layer + ff) + pairs * heads * 4 * 128
        moved = (layer + ff) * size + kv_bytes
        if kind == "dense":
            return {"bytes": moved + 3 * tokens * width * size, "flops": flops}
        rows = case["seqs"]
        return {"bytes": moved * case["layers"] + case["vocab"] * (width * size + rows * 4) + tokens * width * size,
                "flops": flops * case["layers"] + 2 * rows * width * case["vocab"]}
    if kind == "experts":
        inner = width * case["ff"] * (2 if case["expert"] == "relu2" else 3)
        used = case["experts"] * (1.0 - (1.0 - case["top"] / case["experts"]) ** tokens)
        return {"bytes": used * inner * size + 2 * tokens * width * size + case["experts"] * width * 4,
                "flops": 2 * tokens * (case["top"] * inner + case["experts"] * width)}
    if kind == "latent":
        q_rank, rank, row = width * 3 // 4 // 64 * 64, case["rank"], case["rank"] + 64
        matrices = width * (q_rank + row + heads * 128) + q_rank * heads * 192 + 2 * heads * 128 * rank + width * heads * 128
        seen = [_seen(past, new, case["window"]) for past, new in lengths]
        pairs = sum(n for n, _ in seen)
        # scores and sums over the cached latents themselves (what a step of few tokens does), or over keys and values
        # of 192 and 128 a head that are first formed from them (less work for a prompt)
        over_latents = pairs * heads * 2 * (row + rank)
        formed = pairs * heads * 2 * (192 + 128) + 2 * sum(keys for _, keys in seen) * heads * 256 * rank
        return {"bytes": matrices * size + sum(keys for _, keys in seen) * row * size + 2 * tokens * width * size,
                "flops": 2 * tokens * matrices + min(over_latents, formed)}
    if kind == "window":
        matrices = width * 128 * (2 * heads + 2 * groups)
        seen = [_seen(past, new, case["window"]) for past, new in lengths]
        return {"bytes": matrices * size + sum(keys for _, keys in seen) * 2 * groups * 128 * size + 2 * tokens * width * size,
                "flops": 2 * tokens * matrices + sum(n for n, _ in seen) * heads * 4 * 128}
    inner = heads * 128
    matrices = {"state_space": width * (2 * inner + 256 + 2 * heads), "gated_delta": width * (3 * inner + 2 * heads),
                "forget_write": width * 3 * inner, "gated_linear_attention": width * (4 * inner + 16) + 16 * inner}[kind]
    matrices += inner * width
    state = heads * 128 * 128 * 4 * 2 * case["seqs"]
    return {"bytes": matrices * size + state + 2 * tokens * width * size,
            "flops": 2 * tokens * matrices + tokens * heads * 128 * 128 * (6 if kind == "gated_delta" else 4)}


def tolerance(case):
    if case["dtype"] == "fp32":
        return {"rel": 2e-5, "max": 1e-3}
    if case["kind"] == "model":
        # roundings of 16 bits that travel through up to four layers: 0.02 off the same in 64 bits
        return {"rel": 0.03, "max": 0.2}
    # 0.004 to 0.006 off the same in 64 bits
    return {"rel": 0.02, "max": 0.15}


# ------------------------------------------------------------------------------------------ the same in 64 bits

F = torch.float64


def _norm(x, gain, eps):
    y = x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)
    return y if gain is None else y * gain


def _silu(x):
    return x * torch.sigmoid(x)


def _softplus(x):
    return torch.logaddexp(x, torch.zeros_like(x))


def _conv(x, taps, bias=None):
    """A causal convolution per channel: the last tap multiplies the current token."""
    y = torch.zeros_like(x) if bias is None else bias.expand_as(x).clone()
    for back in range(min(taps.shape[1], x.shape[0])):
        y[back:] += taps[:, taps.shape[1] - 1 - back] * x[:x.shape[0] - back]
    return y


def _angles(count, dims, base):
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=F, device=DEVICE) / dims)
    a = torch.arange(count, dtype=F, device=DEVICE)[:, None] * f
    return a.cos()[:, None, :], a.sin()[:, None, :]


def _turn(x, dims, base, interleaved):
    """The first ``dims`` entries of the heads of ``x`` ``[T, heads, D]`` turned by their positions from 0 on."""
    cos, sin = _angles(x.shape[0], dims, base)
    one = slice(0, dims, 2) if interleaved else slice(0, dims // 2)
    two = slice(1, dims, 2) if interleaved else slice(dims // 2, dims)
    out, u, v = x.clone(), x[..., one], x[..., two]
    out[..., one], out[..., two] = u * cos - v * sin, v * cos + u * sin
    return out


def _attend(q, k, v, scale, first, window=0, sink=None, cap=0.0):
    """The queries from position ``first`` on, head by head: ``q`` ``[T, H, D]``, ``k``/``v`` ``[T, G, ...]``."""
    t, heads = q.shape[0], q.shape[1]
    i, j = torch.arange(first, t, device=DEVICE)[:, None], torch.arange(t, device=DEVICE)[None, :]
    hidden = (j > i) | ((i - j >= window) if window else (j > i))
    out = torch.empty((t - first, heads, v.shape[2]), dtype=F, device=DEVICE)
    for h in range(heads):
        g = h // (heads // k.shape[1])
        s = (q[first:, h] @ k[:, g].T) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill_(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(s.shape[0], 1)], dim=1)
        out[:, h] = torch.softmax(s, dim=-1)[:, :t] @ v[:, g]
    return out


def _gated(x, w, gate="gate", up="up", down="down"):
    return (_silu(x @ w[gate].T) * (x @ w[up].T)) @ w[down].T


def _dense_attention(x, w, heads, groups, theta, first, eps=1e-6):
    t = x.shape[0]
    q = _norm((x @ w["q"].T).view(t, heads, 128), w["q_norm"], eps)
    k = _norm((x @ w["k"].T).view(t, groups, 128), w["k_norm"], eps)
    v = (x @ w["v"].T).view(t, groups, 128)
    a = _attend(_turn(q, 128, theta, False), _turn(k, 128, theta, False), v, 128 ** -0.5, first)
    return a.flatten(1) @ w["o"].T


def _recurrence(case, x, w):
    """``(output rows, state [H, N, V])`` of one whole sequence."""
    kind, heads, t = case["kind"], case["heads"], x.shape[0]
    inner = heads * 128
    skip = None
    if kind == "state_space":
        heads = 2 * heads
        p = x @ w["in"].T
        z, xbc, dt = p[:, :inner], p[:, inner:2 * inner + 256], p[:, 2 * inner + 256:]
        xbc = _silu(_conv(xbc, w["conv"], w["conv_bias"]))
        v = xbc[:, :inner].view(t, heads, 64)
        k = xbc[:, None, inner:inner + 128].expand(t, heads, 128)
        q = xbc[:, None, inner + 128:].expand(t, heads, 128)
        dt = _softplus(dt + w["dt_bias"])
        decay = torch.exp(-torch.exp(w["A_log"]) * dt)[:, :, None, None]
        write = dt[:, :, None] * v
        skip = w["D"][:, None] * v
    elif kind == "gated_delta":
        half = heads // 2
        q = _silu(_conv(x @ w["q"].T, w["q_conv"])).view(t, half, 128)
        k = _silu(_conv(x @ w["k"].T, w["k_conv"])).view(t, half, 128)
        v = _silu(_conv(x @ w["v"].T, w["v_conv"])).view(t, heads, 128)
        q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * 128 ** -0.5).repeat_interleave(2, dim=1)
        k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(2, dim=1)
        beta = torch.sigmoid(x @ w["b"].T)[:, :, None]
        decay = torch.exp(-torch.exp(w["A_log"]) * _softplus(x @ w["a"].T + w["dt_bias"]))[:, :, None, None]
        write = v
    else:
        v = (x @ w["v"].T).view(t, heads, 128)
        q = (x @ w["q"].T).view(t, heads, 128)
        if kind == "forget_write":
            q = _silu(q)
            f = w["lower"] + (1.0 - w["lower"]) * torch.sigmoid(x @ w["f"].T + w["f_bias"])
            decay = f.view(t, heads, 128)[..., None]
            k = 1.0 - decay[..., 0]
        else:
            q = q * 128 ** -0.5
            k = (x @ w["k"].T).view(t, heads, 128)
            f = (x @ w["a1"].T) @ w["a2"].T + w["a2_bias"]
            decay = torch.exp(torch.nn.functional.logsigmoid(f) / 16.0).view(t, heads, 128)[..., None]
        write = v
    state = torch.zeros((heads, 128, v.shape[2]), dtype=F, device=DEVICE)
    out = torch.empty_like(v)
    for i in range(t):
        state = decay[i] * state
        u = write[i]
        if kind == "gated_delta":
            u = beta[i] * (u - (k[i][:, None, :] @ state)[:, 0])
        state = torch.addcmul(state, k[i][:, :, None], u[:, None, :])
        out[i] = (q[i][:, None, :] @ state)[:, 0]
    if kind == "state_space":
        o = _norm((out + skip).reshape(t, inner) * _silu(z), w["norm"], 1e-6)
    else:
        o = _norm(out, w["norm"], 1e-6).reshape(t, inner)
        if kind != "forget_write":
            o = o * _silu(x @ w["g"].T)
    return o @ w["o"].T, state


def _mix(case, x, w, first):
    """The mixer of a case on one whole sequence: the rows from ``first`` on."""
    t, heads, groups = x.shape[0], case["heads"], case["kv_heads"]
    if case["kind"] == "dense":
        return _dense_attention(x, w, heads, groups, 1e6, first)
    if case["kind"] == "latent":
        rank = case["rank"]
        q = (_norm(x @ w["dq"].T, w["dq_norm"], 1e-6) @ w["uq"].T).view(t, heads, 192)
        q = torch.cat([q[..., :128], _turn(q[..., 128:], 64, 1e4, True)], dim=-1)
        down = x @ w["dkv"].T
        c = _norm(down[:, :rank], w["dkv_norm"], 1e-6)
        shared = _turn(down[:, None, rank:], 64, 1e4, True)
        k = torch.cat([(c @ w["uk"].T).view(t, heads, 128), shared.expand(t, heads, 64)], dim=-1)
        v = (c @ w["uv"].T).view(t, heads, 128)
        a = _attend(q, k, v, 192 ** -0.5, first, case["window"], w.get("sink"))
        return (a.flatten(1) * torch.sigmoid(x[first:] @ w["g"].T)) @ w["o"].T

    def project(name):
        return _conv(x @ w[name].T + w[name + "_bias"], w[name + "_conv"])

    q = _norm(project("q"), w["q_norm"], 1e-6).view(t, heads, 128)
    k = _norm(project("k"), w["k_norm"], 1e-6).view(t, groups, 128)
    v = project("v").view(t, groups, 128)
    a = _attend(_turn(q, 128, 1e6, True), _turn(k, 128, 1e6, True), v, 128 ** -0.5, first, case["window"], w.get("sink"), case["cap"])
    return a.flatten(1) @ w["o"].T


def _experts(case, x, w):
    scores = x @ w["router"].T
    if case["expert"] == "gated_clamped":
        scores = scores + w["router_bias"]
    best, ids = torch.topk(scores, case["top"], dim=-1)
    if case["expert"] == "gated_clamped":
        weight = torch.softmax(best, dim=-1)
    else:
        weight = torch.sigmoid(best)
        if case["expert"] == "relu2":
            weight = weight / (weight.sum(-1, keepdim=True) + 1e-20) * 2.5
    out = torch.zeros_like(x)
    for e in range(case["experts"]):
        row, place = torch.nonzero(ids == e, as_tuple=True)
        h, up, down = x[row], w[f"e{e}_up"].to(F), w[f"e{e}_down"].to(F)
        if case["expert"] == "relu2":
            a = torch.relu(h @ up.T) ** 2
        else:
            g, u = h @ w[f"e{e}_gate"].to(F).T, h @ up.T
            if case["expert"] == "gated_silu":
                a = _silu(g) * u
            else:
                g = g.clamp(max=7.0)
                a = g * torch.sigmoid(1.702 * g) * (u.clamp(-7.0, 7.0) + 1.0)
        out.index_add_(0, row, weight[row, place, None] * (a @ down.T))
    return out


@torch.no_grad()
def exact(case, seed):
    if case["kind"] == "model":
        return {"logits": _exact_model(case, seed)}
    _, weights = _parts(case, seed)
    weights = [{n: v if n[0] == "e" and n[1].isdigit() else v.to(F) for n, v in w.items()} for w in weights]
    ys, states = [], []
    rows = _inputs(case, seed)
    new = torch.cat([b for _, b in rows]).to(F)
    if case["kind"] == "experts":
        return {"y0": _experts(case, new, weights[0])}
    out = {}
    for past, step in rows:
        x = torch.cat([past, step]).to(F)
        if case["kind"] in RECURRENT:
            y, last = _recurrence(case, x, weights[0])
            ys.append(y[past.shape[0]:])
            states.append(last)
        else:
            ys.append(_mix(case, x, weights[0], past.shape[0]))
    out["y0"] = torch.cat(ys)
    if case["kind"] == "dense":
        out["y1"] = _gated(new, weights[1])
    if states:
        out["recurrent"] = torch.stack(states)
    return out


def _exact_model(case, seed):
    model = random_model(_model_config(case), seed, DTYPES[case["dtype"]], DEVICE)
    drawn = random_checkpoint(model.expected_tensors(), seed, DTYPES[case["dtype"]], DEVICE)
    names = {"q": "self_attn.q_proj", "k": "self_attn.k_proj", "v": "self_attn.v_proj", "o": "self_attn.o_proj",
             "q_norm": "self_attn.q_norm", "k_norm": "self_attn.k_norm", "norm1": "input_layernorm",
             "norm2": "post_attention_layernorm", "gate": "mlp.gate_proj", "up": "mlp.up_proj", "down": "mlp.down_proj"}
    embed = drawn["model.embed_tokens.weight"]
    sequences = [embed[torch.tensor(seq, device=DEVICE)].to(F) for seq in _tokens(case, seed)]
    for i in range(case["layers"]):
        w = {short: drawn[f"model.layers.{i}.{name}.weight"].to(F) for short, name in names.items()}
        for n, x in enumerate(sequences):
            x = x + _dense_attention(_norm(x, w["norm1"], 1e-6), w, case["heads"], case["kv_heads"], 5e6, 0)
            sequences[n] = x + _gated(_norm(x, w["norm2"], 1e-6), w)
    last = _norm(torch.stack([x[-1] for x in sequences]), drawn["model.norm.weight"].to(F), 1e-6)
    return torch.cat([last @ part.to(F).T for part in embed.split(16384)], dim=1)
