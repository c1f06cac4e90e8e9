"""The work this engine is measured on: its layers over prompts and over single tokens, a batch served from prompt to
generated tokens, and the choice of the next token.

A mixer or feed-forward is built from its part specification, is given a step's description and its cache, and runs one
step, as the step function runs it; ``serve`` goes through the step function itself, ``sample`` through the sampler.
Layer sizes are those of ``bench.py`` and the ``bench_*`` files (width 2,048 or 4,096); weights are random with the
spread a checkpoint has, decays and step sizes spread as in trained recurrent layers (memories of a few to a few
thousand tokens).

A case: ``kind``, ``width``, ``rows`` (requests in the step), ``tokens`` (of all rows; as many as rows: single tokens), ``context``
(positions a row already holds in its cache or state; rows differ), ``dtype``.
"""

from __future__ import annotations

import math

import torch

from kairyu_b200.cache.manager import CacheLayout, CacheManager
from kairyu_b200.cache.storage import CacheStorage
from kairyu_b200.engine.engine import build_model
from kairyu_b200.engine.runner import ModelRunner, StepEntry
from kairyu_b200.engine.workspace import Workspace
from kairyu_b200.parts.base import FEED_FORWARDS, MIXERS, PartSpec, StepContext
from kairyu_b200.sampling.params import SamplingParams
from kairyu_b200.sampling.sampler import Sampler, SamplingRow

PAGE = 16
EPS = 1e-5
THETA = 500000.0
POSITIONS = 8192
VOCAB = 32000
SAMPLE_VOCAB = 128256
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
DEVICE = "cuda"


def _case(kind, name=None, *, width=2048, rows=1, tokens=1, context=0, dtype="bfloat16", **more):
    case = {"kind": kind, "width": width, "rows": rows, "tokens": tokens, "context": context, "dtype": dtype, **more}
    return dict(case, name=name) if name else case


def listed():
    return [
        # eight requests answered from prompt to 32 generated tokens by a dense decoder of eight layers: the whole engine below the scheduler
        _case("serve", "serve dense 8 requests", rows=8, tokens=2000, steps=32),
        # a portion of a long prompt beside decoded tokens, as chunked prefill runs it, at the Llama-3.1-8B layer sizes
        _case("gqa", "attention portion beside decodes", width=4096, rows=7, tokens=518, context=3500),
        # the 32-bit mode, in which results do not depend on how prompts were cut: three prompts of a few hundred tokens
        _case("gqa", "attention 32-bit 3 prompts", rows=3, tokens=700, dtype="float32"),
        # recurrent layers over one prompt (nothing but the prompt's own length to spread over the device)
        _case("delta", "delta rule prompt 2048", tokens=2048),
        # ... and over a batch of prompts of unequal lengths, some of them continuing, with a decay a key channel
        _case("delta", "delta rule channel 6 prompts", width=4096, rows=6, tokens=5001, context=700, channel=True),
        _case("ssm", "state space prompt 2048", tokens=2048),
        # differential attention over a prompt, and over a batch of decoded tokens
        _case("diff", "differential prompt 2048", tokens=2048),
        _case("diff", "differential decode 64", rows=64, tokens=64, context=2000),
        # latent attention with a rotated key part and an output gate: the rows are 256 columns wide
        _case("latent", "latent prompts 2048", rows=3, tokens=2048, context=900),
        # a mixture of experts for a decode step and for a prompt
        _case("moe", "experts decode 8", rows=8, tokens=8),
        _case("moe", "experts prompt 2048", tokens=2048),
        # the next token of a small batch with the filters chat requests use, with a report of log-probabilities
        _case("sample", "sample 8", width=SAMPLE_VOCAB, rows=8, tokens=8),
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["serve", "gqa", "gqa", "delta", "delta", "ssm", "ssm", "diff", "diff", "latent", "moe", "moe", "sample"])
    if kind == "serve":
        rows = _spread(rng, 1, 16)
        return _case(kind, rows=rows, tokens=max(rows * 2, _spread(rng, 40, 2000)), steps=_spread(rng, 4, 28))
    if kind == "sample":
        rows = _spread(rng, 1, 64)
        return _case(kind, width=SAMPLE_VOCAB, rows=rows, tokens=rows)
    width = rng.choice([2048, 2048, 4096])
    if rng.random() < 0.35:  # a decode step
        rows = _spread(rng, 1, 128)
        tokens = rows
    else:
        tokens = _spread(rng, 17, 5000 if kind in ("delta", "ssm") else 2500)
        rows = min(tokens // 8 + 1, _spread(rng, 1, 12))
    context = rng.choice([0, _spread(rng, 20, 3000)]) if tokens > rows else _spread(rng, 20, 2500)
    more = {}
    dtype = "bfloat16"
    if kind == "delta":
        more["channel"] = rng.random() < 0.5
    if kind in ("gqa", "delta", "ssm") and rng.random() < 0.2:
        dtype, width, tokens = "float32", 2048, min(tokens, 900 + rows)
    if kind == "moe":
        context, width, tokens = 0, 2048, min(tokens, 2048)
        rows = min(rows, tokens)
    return _case(kind, width=width, rows=rows, tokens=tokens, context=context, dtype=dtype, **more)


# ------------------------------------------------------------------ sizes


def _counts(case):
    """Tokens of each row: single tokens where there are as many rows as tokens; the gqa kind puts one portion beside
    decoded tokens when its rows are few beside its tokens; otherwise unequal prompts."""
    rows, tokens = case["rows"], case["tokens"]
    if rows == tokens:
        return [1] * rows
    if case["kind"] == "gqa" and rows > 4:
        return [tokens - (rows - 1)] + [1] * (rows - 1)
    shares = [1.0 + 0.7 * math.sin(2.3 * i + 0.4) for i in range(rows)]
    counts = [max(1, int(tokens * s / sum(shares))) for s in shares]
    counts[0] += tokens - sum(counts)
    return counts


def _contexts(case):
    """Positions each row holds already; of several prompts every third is new."""
    context = case["context"]
    return [0 if n > 1 and i % 3 == 2 else max(0, context - 37 * i % (context // 2 + 1)) for i, n in enumerate(_counts(case))]


def _sizes(case):
    width = case["width"]
    heads = width // 128
    kind = case["kind"]
    if kind == "gqa":
        return dict(heads=heads, kv=max(heads // 4, 1), dim=128)
    if kind == "delta":
        return dict(heads=heads, kv=heads // 2, dim=128, vdim=128, taps=4, rank=64)
    if kind == "ssm":
        return dict(heads=2 * width // 64, vdim=64, state=128, groups=8, taps=4)
    if kind == "diff":
        return dict(heads=heads, kv=heads // 4, dim=64, vdim=128, window=1024, softcap=50.0, lam_init=0.4)
    if kind == "latent":
        return dict(heads=heads, dim=128, rot=64, vdim=128, rank=192)
    if kind == "moe":
        return dict(experts=32, top=4, ff=1024, limit=7.0, alpha=1.702, shift=1.0)
    return {}


def _rope_spec(dims):
    return PartSpec("rope", rotary_dim=dims, theta=THETA, scaling=None, max_positions=POSITIONS, wide_angles=True)


def _part_spec(case):
    s, width = _sizes(case), case["width"]
    kind = case["kind"]
    if kind == "gqa":
        return PartSpec("gqa_attention", prefix="m", hidden_size=width, num_heads=s["heads"], num_kv_heads=s["kv"], head_dim=128, qk_norm=False,
                        norm_eps=EPS, qkv_bias=False, o_bias=False, position=_rope_spec(128))
    if kind == "delta":
        more = dict(decay="channel", decay_rank=s["rank"], gate_rank=s["rank"], gate_activation="sigmoid") if case.get("channel") else {}
        return PartSpec("gated_delta", prefix="m", hidden_size=width, num_heads=s["heads"], num_kv_heads=s["kv"], head_dim=s["dim"],
                        value_dim=s["vdim"], conv_taps=s["taps"], norm_eps=EPS, **more)
    if kind == "ssm":
        return PartSpec("state_space_dual", prefix="m", hidden_size=width, num_heads=s["heads"], value_dim=s["vdim"], state_size=s["state"],
                        groups=s["groups"], norm_groups=s["groups"], conv_taps=s["taps"], norm_eps=EPS)
    if kind == "diff":
        return PartSpec("differential_attention", prefix="m", hidden_size=width, num_heads=s["heads"], num_kv_heads=s["kv"], head_dim=s["dim"],
                        value_dim=s["vdim"], scale=s["dim"] ** -0.5, lam_init=s["lam_init"], norm_eps=EPS, softcap=s["softcap"], window=s["window"],
                        keep=s["window"])
    if kind == "latent":
        return PartSpec("latent_attention", prefix="m", hidden_size=width, num_heads=s["heads"], head_dim=s["dim"], value_dim=s["vdim"], kv_rank=s["rank"],
                        scale=(s["dim"] + s["rot"]) ** -0.5, norm_eps=EPS, rot_dim=s["rot"], position=_rope_spec(s["rot"]), rotary_interleaved=False, gate=True)
    return PartSpec("moe", prefix="m", hidden_size=width, intermediate_size=s["ff"], num_experts=s["experts"], top=s["top"], limit=s["limit"],
                    alpha=s["alpha"], shift=s["shift"])


# ------------------------------------------------------------------ inputs


def _generator(seed, what):
    g = torch.Generator(device=DEVICE)
    g.manual_seed((int(seed) * 7919 + what) & 0x7FFFFFFF)
    return g


def _weights(specs, dtype, seed):
    """One tensor a name; spread as in a checkpoint."""
    held = {}
    for index, spec in enumerate(specs):
        if spec.alias_of is not None:
            continue
        g = _generator(seed, 1000 + index)
        last = spec.name.split(".")[-1]
        if last == "A_log":    # rates of 1 to 16
            t = torch.log(1.0 + 15.0 * torch.rand(spec.shape, generator=g, device=DEVICE))
        elif last == "dt_bias":  # softplus of it: steps of 0.001 to 0.1
            step = torch.exp(math.log(1e-3) + (math.log(0.1) - math.log(1e-3)) * torch.rand(spec.shape, generator=g, device=DEVICE))
            t = step + torch.log(-torch.expm1(-step))
        elif last == "conv" or spec.init == "taps":
            t = torch.rand(spec.shape, generator=g, device=DEVICE) - 0.5
        elif spec.init == "norm":
            t = 1.0 + 0.1 * torch.randn(spec.shape, generator=g, device=DEVICE)
        else:
            t = 0.02 * torch.randn(spec.shape, generator=g, device=DEVICE)
        held[spec.name] = t.to(dtype) if spec.role == "matrix" else t.float()
    return held


def _pages(case, seed):
    """Per row its physical pages (shuffled; page 0 is the pool's reserved one), and how many there are."""
    lengths = [c + n for c, n in zip(_contexts(case), _counts(case))]
    need = [-(-length // PAGE) for length in lengths]
    order = (torch.randperm(sum(need), generator=torch.Generator().manual_seed(int(seed))) + 1).tolist()
    tables, at = [], 0
    for n in need:
        tables.append(order[at : at + n])
        at += n
    return tables, sum(need) + 1


def _rows_in(case, seed):
    x = torch.randn((case["tokens"], case["width"]), generator=_generator(seed, 1), device=DEVICE)
    return x.to(DTYPES[case["dtype"]])


def _int32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEVICE)


def _step(case, part, tables, dtype):
    counts, contexts = _counts(case), _contexts(case)
    starts = [0]
    for n in counts:
        starts.append(starts[-1] + n)
    lengths = [c + n for c, n in zip(contexts, counts)]
    singles = [row for row, n in enumerate(counts) if n == 1]
    tiles = {}
    for size in getattr(part, "query_tile_sizes", lambda: ())():
        at = [(row, first) for row, n in enumerate(counts) if n > 1 for first in range(0, n, size)]
        tiles[size] = (len(at), _int32([row for row, _ in at]), _int32([first for _, first in at]))
    width = max((len(t) for t in tables), default=1)
    block_table = _int32([t + [-1] * (width - len(t)) for t in tables])
    return StepContext(
        num_tokens=starts[-1], num_rows=len(counts), dtype=dtype, token_ids=torch.zeros(starts[-1], dtype=torch.int32, device=DEVICE),
        positions=torch.cat([torch.arange(c, c + n, dtype=torch.int32, device=DEVICE) for c, n in zip(contexts, counts)]),
        row_ids=_int32([row for row, n in enumerate(counts) for _ in range(n)]), qo_indptr=_int32(starts), seq_lens=_int32(lengths),
        write_from=torch.zeros(len(counts), dtype=torch.int32, device=DEVICE), state_slots=torch.arange(len(counts), dtype=torch.int32, device=DEVICE),
        block_tables={0: block_table}, host_qo_indptr=tuple(starts), host_seq_lens=tuple(lengths), tiles=tiles, num_decode_rows=len(singles),
        decode_rows=_int32(singles), decode_tokens=_int32([starts[row] for row in singles]), max_seq_len=max(lengths),
        max_portion_seq_len=max((length for length, n in zip(lengths, counts) if n > 1), default=0), workspace=Workspace(DEVICE),
        error_flag=torch.zeros(1, dtype=torch.int32, device=DEVICE),
    )


def _cache(case, part, num_pages, dtype, seed):
    """The cache as earlier steps left it: rows of unit spread in the pages, a filled memory for rows with a context."""
    layout = CacheLayout.from_slot_specs({0: tuple(part.cache_specs())})
    storage = CacheStorage(layout, num_pages=num_pages, page_size=PAGE, max_requests=case["rows"], dtype=dtype, device=DEVICE)
    for index, tensor in enumerate([*storage.k, *storage.v]):
        if tensor.numel():
            tensor.copy_(torch.randn(tensor.shape, generator=_generator(seed, 100 + index), device=DEVICE))
    for index, tensor in enumerate(storage.states):
        tensor.copy_((0.1 if index == 0 else 1.0) * torch.randn(tensor.shape, generator=_generator(seed, 200 + index), device=DEVICE))
        for row, context in enumerate(_contexts(case)):
            if context == 0:
                tensor[row].zero_()
    return storage


def _dense_config(case):
    width = case["width"]
    return {"architectures": ["LlamaForCausalLM"], "hidden_size": width, "num_hidden_layers": 8, "num_attention_heads": width // 128,
            "num_key_value_heads": width // 512, "head_dim": 128, "intermediate_size": 4 * width, "vocab_size": VOCAB, "rope_theta": THETA,
            "max_position_embeddings": POSITIONS, "rms_norm_eps": EPS, "tie_word_embeddings": False, "hidden_act": "silu"}


def _dialogue(case, seed):
    """Per row its prompt and the tokens that follow it."""
    g = torch.Generator().manual_seed(int(seed))
    return [(torch.randint(0, VOCAB, (n,), generator=g).tolist(), torch.randint(0, VOCAB, (case["steps"],), generator=g).tolist()) for n in _counts(case)]


def _logits(case, seed):
    """Next-token logits of a language model's spread: most of the mass on a few dozen tokens."""
    g = _generator(seed, 1)
    z = 2.0 * torch.randn((case["rows"], case["width"]), generator=g, device=DEVICE)
    places = torch.randint(0, case["width"], (case["rows"], 64), generator=g, device=DEVICE)
    return z.scatter_(1, places, 9.0 + 2.0 * torch.randn((case["rows"], 64), generator=g, device=DEVICE))


def prepare(case, seed):
    dtype = DTYPES[case["dtype"]]
    if case["kind"] == "sample":
        rows = [SamplingRow(request_id=f"r{i}", position=11 + i, params=SamplingParams(
            temperature=0.0 if i % 8 == 7 else 0.8, top_p=0.9 if i % 3 else 1.0, top_k=50 if i % 2 else -1, min_p=0.02 if i % 5 == 4 else 0.0, logprobs=5,
            seed=int(seed) + i)) for i in range(case["rows"])]
        return {"kind": "sample", "logits": _logits(case, seed), "rows": rows, "sampler": Sampler(case["width"], DEVICE)}
    if case["kind"] == "serve":
        model, _ = build_model(_dense_config(case), dtype=case["dtype"], device=DEVICE)
        model.load(_weights(model.tensor_specs(), dtype, seed))
        longest = max(_counts(case)) + case["steps"]
        pages = sum(-(-(n + case["steps"]) // PAGE) for n in _counts(case)) + 1
        layout = CacheLayout.from_slot_specs(model.cache_slot_specs())
        cache = CacheManager(layout, num_pages=pages, page_size=PAGE, max_requests=case["rows"])
        storage = CacheStorage(layout, num_pages=pages, page_size=PAGE, max_requests=case["rows"], dtype=dtype, device=DEVICE)
        runner = ModelRunner(model, cache, storage, max_model_len=longest, decode_mode="cuda_graph", max_graph_batch=case["rows"])
        for length in (longest, min(_counts(case)) + 1):
            runner.capture_decode_graphs(case["rows"], length)
        return {"kind": "serve", "runner": runner, "dialogue": _dialogue(case, seed), "steps": case["steps"]}
    registry = FEED_FORWARDS if case["kind"] == "moe" else MIXERS
    part = registry.build(_part_spec(case), dtype=dtype, device=DEVICE, shared={})
    part.load(_weights(part.tensor_specs(), dtype, seed))
    state = {"kind": case["kind"], "part": part, "x": _rows_in(case, seed)}
    if case["kind"] == "moe":
        return dict(state, ctx=_step(case, part, [[1]] * case["rows"], dtype))
    tables, pages = _pages(case, seed)
    storage = _cache(case, part, pages, dtype, seed)
    return dict(state, ctx=_step(case, part, tables, dtype), cache=storage.view(0, writes=True), states=storage.states)


# ------------------------------------------------------------------ the pass


def run(state):
    kind = state["kind"]
    if kind == "sample":
        ids = state["sampler"].sample(state["logits"], state["rows"])
        report = state["sampler"].take_report()
        return {"ids": ids, "chosen": report.values[:, 0], "top": report.values[:, 1:], "top_ids": report.indices}
    if kind == "serve":
        return _serve(state)
    if kind == "moe":
        return {"out": state["part"].forward(state["x"], state["ctx"])}
    out = state["part"].forward(state["x"], state["ctx"], state["cache"])
    if not state["states"]:
        return {"out": out}
    return {"out": out, "memory": state["states"][0][:-1]}


def _serve(state):
    runner, dialogue = state["runner"], state["dialogue"]
    names = [f"r{i}" for i in range(len(dialogue))]
    logits = [runner.step([StepEntry(name, prompt, (len(prompt) - 1,)) for name, (prompt, _) in zip(names, dialogue)]).clone()]
    for step in range(state["steps"]):
        entries = [StepEntry(name, [told[step]], (0,)) for name, (_, told) in zip(names, dialogue)]
        logits.append(runner.step(entries).clone())
    for name in names:
        runner.cache.release(name)
    return torch.stack(logits)


# ------------------------------------------------------------------ what a pass cannot do without


def _seen(case, window=None):
    """Keys seen, summed over the step's tokens, and positions read, summed over its rows."""
    pairs = positions = 0
    for c, n in zip(_contexts(case), _counts(case)):
        if window is None:
            pairs += n * c + n * (n + 1) // 2
            positions += c + n
        else:
            pairs += sum(min(window, c + i + 1) for i in range(n))
            positions += min(c + n, n + window - 1)
    return pairs, positions


def work(case):
    kind, width, T, R = case["kind"], case["width"], case["tokens"], case["rows"]
    e = 2 if case["dtype"] == "bfloat16" else 4
    s = _sizes(case)
    if kind == "sample":
        return {"bytes": 4 * R * width, "flops": 8 * R * width}
    if kind == "serve":
        layer = width * (width + 2 * (width // 4)) + width * width + 3 * width * 4 * width
        head = width * VOCAB
        pairs = positions = 0
        for n in _counts(case):
            pairs += sum(range(1, n + case["steps"] + 1))
            positions += sum(range(n, n + case["steps"] + 1))
        every = T + R * case["steps"]
        wanted = R * (case["steps"] + 1)
        return {"bytes": e * ((case["steps"] + 1) * (8 * layer + head) + 8 * 2 * (width // 4) * positions) + 4 * VOCAB * wanted,
                "flops": 2 * (8 * layer * every + head * wanted) + 8 * 4 * pairs * width}
    if kind == "moe":
        touched = s["experts"] * (1 - (1 - s["top"] / s["experts"]) ** T)
        return {"bytes": e * (touched * 3 * width * s["ff"] + 2 * T * width), "flops": 2 * T * s["top"] * 3 * width * s["ff"] + 2 * T * width * s["experts"]}
    if kind == "gqa":
        rows = s["heads"] * 128 + 2 * s["kv"] * 128
        pairs, positions = _seen(case)
        weights = width * (rows + s["heads"] * 128)
        return {"bytes": e * (weights + 2 * T * width + 2 * s["kv"] * 128 * positions), "flops": 2 * T * weights + 4 * pairs * s["heads"] * 128}
    if kind == "diff":
        rows = s["heads"] * 2 * s["dim"] + s["kv"] * (2 * s["dim"] + s["vdim"])
        pairs, positions = _seen(case, s["window"])
        weights = width * (rows + s["heads"] * s["vdim"])
        return {"bytes": e * (weights + 2 * T * width + s["kv"] * (2 * s["dim"] + s["vdim"]) * positions),
                "flops": 2 * T * weights + 2 * pairs * s["heads"] * 2 * (s["dim"] + s["vdim"])}
    if kind == "latent":
        row = s["rank"] + s["rot"]
        pairs, positions = _seen(case)
        weights = width * (s["heads"] * (s["dim"] + s["rot"]) + row + 2 * s["heads"] * s["vdim"]) + s["heads"] * s["rank"] * (s["dim"] + s["vdim"])
        return {"bytes": e * (weights + 2 * T * width + row * positions), "flops": 2 * T * weights + 2 * pairs * s["heads"] * (row + s["rank"])}
    if kind == "delta":
        q, v = s["kv"] * s["dim"], s["heads"] * s["vdim"]
        if case.get("channel"):
            weights = width * (2 * q + 2 * v + s["heads"] + 2 * s["rank"]) + s["rank"] * (s["heads"] * s["dim"] + v)
        else:
            weights = width * (2 * q + 3 * v + 2 * s["heads"])
        memory = s["heads"] * s["dim"] * s["vdim"]
        return {"bytes": e * (weights + 2 * T * width) + 8 * R * memory, "flops": 2 * T * weights + 6 * T * memory}
    inner, bc = s["heads"] * s["vdim"], s["groups"] * s["state"]
    weights = width * (3 * inner + 2 * bc + s["heads"])
    memory = s["heads"] * s["vdim"] * s["state"]
    return {"bytes": e * (weights + 2 * T * width) + 8 * R * memory, "flops": 2 * T * weights + 4 * T * memory}


def tolerance(case):
    """Four times what a path shows against its result in 64 bits: the roundings of 16-bit activations between a layer's kernels, or
    32-bit sums in another order."""
    if case["kind"] == "sample":  # a draw may fall the other way where two noisy logits are equal to the last bit
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    if case["kind"] == "serve":
        return {"rel": 0.03, "max": 0.3}
    return {"rel": 0.015, "max": 0.3}


# ------------------------------------------------------------------ the same in 64 bits


def _turn(x, positions, dims):
    """Pairs (i, i + dims/2) of the last dimension turned by position * theta^(-2i/dims); x [tokens, heads, dims]."""
    half = dims // 2
    f = THETA ** (-torch.arange(half, dtype=torch.float64, device=x.device) * 2 / dims)
    angle = positions.double()[:, None] * f
    cos, sin = angle.cos()[:, None, :], angle.sin()[:, None, :]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)


def _attend(q, k, v, first, scale, window=None, softcap=None):
    """q [n, H, d], k [S, G, d], v [S, G, e]; query i stands at position first + i."""
    n, heads, _ = q.shape
    group = heads // k.shape[1]
    at = torch.arange(n, device=q.device)[:, None] + first
    key = torch.arange(k.shape[0], device=q.device)[None, :]
    hidden = (key > at) | ((key <= at - window) if window else torch.zeros_like(key > at))
    out = []
    for h in range(heads):
        s = (q[:, h] @ k[:, h // group].T) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        out.append(torch.softmax(s.masked_fill(hidden, -math.inf), dim=-1) @ v[:, h // group])
    return torch.stack(out, dim=1)


def _paged(storage, tables, row, length, index):
    pages = storage[index][0][torch.tensor(tables[row], device=DEVICE)]
    return pages.reshape(-1, *pages.shape[2:])[:length].double()


def _silu(z):
    return z * torch.sigmoid(z)


def _convolve(z, kept, taps):
    """Causal convolution over time a channel: z [n, C], kept [taps - 1, C] inputs before it, taps [C, m] oldest first."""
    every = torch.cat([kept, z])
    m = taps.shape[1]
    return sum(every[j : j + z.shape[0]] * taps[:, j] for j in range(m))


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "sample":
            z = torch.log_softmax(_logits(case, seed).double(), dim=-1)
            return {"ids": None, "chosen": None, "top": torch.topk(z, 5, dim=-1).values, "top_ids": None}
        if kind == "serve":
            return _exact_serve(case, seed)
        dtype = DTYPES[case["dtype"]]
        registry = FEED_FORWARDS if kind == "moe" else MIXERS
        part = registry.build(_part_spec(case), dtype=dtype, device=DEVICE, shared={})  # for the tensors' names and the cache's shapes
        w = {name[2:]: t.double() for name, t in _weights(part.tensor_specs(), dtype, seed).items()}
        x = _rows_in(case, seed).double()
        if kind == "moe":
            return {"out": _exact_moe(case, w, x)}
        tables, pages = _pages(case, seed)
        storage = _cache(case, part, pages, dtype, seed)
        each = {"gqa": _exact_gqa, "diff": _exact_diff, "latent": _exact_latent, "delta": _exact_delta, "ssm": _exact_ssm}[kind]
        outs, memories, at = [], [], 0
        for row, (c, n) in enumerate(zip(_contexts(case), _counts(case))):
            out, memory = each(case, w, x[at : at + n], c, row, tables, storage)
            outs.append(out)
            memories.append(memory)
            at += n
        if memories[0] is None:
            return {"out": torch.cat(outs)}
        return {"out": torch.cat(outs), "memory": torch.stack(memories)}


def _exact_gqa(case, w, x, c, row, tables, storage):
    s, n = _sizes(case), x.shape[0]
    at = torch.arange(c, c + n, device=DEVICE)
    q = _turn((x @ w["q_proj.weight"].T).view(n, s["heads"], 128), at, 128)
    k = _turn((x @ w["k_proj.weight"].T).view(n, s["kv"], 128), at, 128)
    v = (x @ w["v_proj.weight"].T).view(n, s["kv"], 128)
    k = torch.cat([_paged(storage.k, tables, row, c, 0), k])
    v = torch.cat([_paged(storage.v, tables, row, c, 0), v])
    return _attend(q, k, v, c, 128 ** -0.5).reshape(n, -1) @ w["o_proj.weight"].T, None


def _exact_diff(case, w, x, c, row, tables, storage):
    s, n, d = _sizes(case), x.shape[0], _sizes(case)["dim"]
    q = (x @ w["q"].T).view(n, s["heads"], 2, d)
    k = torch.cat([_paged(storage.k, tables, row, c, 0), (x @ w["k"].T).view(n, s["kv"], 2 * d)]).view(c + n, s["kv"], 2, d)
    v = torch.cat([_paged(storage.v, tables, row, c, 0), (x @ w["v"].T).view(n, s["kv"], s["vdim"])])
    lam = torch.exp(w["lq1"] @ w["lk1"]) - torch.exp(w["lq2"] @ w["lk2"]) + s["lam_init"]
    first, second = (_attend(q[:, :, m], k[:, :, m], v, c, d ** -0.5, s["window"], s["softcap"]) for m in (0, 1))
    o = first - lam * second
    o = o * torch.rsqrt(o.square().mean(-1, keepdim=True) + EPS) * (1.0 - s["lam_init"])
    return o.reshape(n, -1) @ w["o"].T, None


def _exact_latent(case, w, x, c, row, tables, storage):
    s, n = _sizes(case), x.shape[0]
    heads, d, rot, rank = s["heads"], s["dim"], s["rot"], s["rank"]
    at = torch.arange(c, c + n, device=DEVICE)
    q = (x @ w["q"].T).view(n, heads, d + rot)
    down = x @ w["dkv"].T
    latent = down[:, :rank] * torch.rsqrt(down[:, :rank].square().mean(-1, keepdim=True) + EPS) * w["dkv.norm"]
    rows = torch.cat([latent, _turn(down[:, None, rank:], at, rot)[:, 0]], dim=1)
    rows = torch.cat([_paged(storage.k, tables, row, c, 0).view(c, rank + rot), rows])
    q_turned = _turn(q[..., d:], at, rot)
    up_k, up_v = w["uk"].view(heads, d, rank), w["uv"].view(heads, s["vdim"], rank)
    q_row = torch.cat([torch.einsum("nhd,hdr->nhr", q[..., :d], up_k), q_turned], dim=-1)
    mixed = _attend(q_row, rows[:, None], rows[:, None, :rank], c, (d + rot) ** -0.5)
    values = torch.einsum("nhr,hvr->nhv", mixed, up_v).reshape(n, -1)
    return (values * torch.sigmoid(x @ w["g"].T)) @ w["o"].T, None


def _exact_delta(case, w, x, c, row, tables, storage):
    s, n = _sizes(case), x.shape[0]
    H, G, D, V = s["heads"], s["kv"], s["dim"], s["vdim"]
    taps = torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]])
    z = torch.cat([x @ w["q"].T, x @ w["k"].T, x @ w["v"].T], dim=1)
    z = _silu(_convolve(z, storage.states[1][row].double(), taps))
    q, k, v = z[:, : G * D].view(n, G, D), z[:, G * D : 2 * G * D].view(n, G, D), z[:, 2 * G * D :].view(n, H, V)
    q = q * torch.rsqrt(q.square().sum(-1, keepdim=True) + 1e-6) * D ** -0.5
    k = k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)
    q, k = q.repeat_interleave(H // G, dim=1), k.repeat_interleave(H // G, dim=1)
    beta = torch.sigmoid(x @ w["b"].T)
    if case.get("channel"):
        a = ((x @ w["a1"].T) @ w["a2"].T + w["dt_bias"]).view(n, H, D)
        g = torch.exp(-torch.exp(w["A_log"])[None, :, None] * torch.nn.functional.softplus(a))
        gate = torch.sigmoid((x @ w["g1"].T) @ w["g2"].T)
    else:
        g = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(x @ w["a"].T + w["dt_bias"]))[..., None].expand(n, H, D)
        gate = _silu(x @ w["g"].T)
    S = storage.states[0][row].double().transpose(1, 2).contiguous()  # [H, D, V]
    outs = []
    for t in range(n):
        S = S * g[t][:, :, None]
        u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
        S = S + k[t][:, :, None] * u[:, None]
        outs.append(torch.bmm(q[t][:, None], S)[:, 0])
    o = torch.stack(outs)
    o = o * torch.rsqrt(o.square().mean(-1, keepdim=True) + EPS) * w["norm"]
    return (o.reshape(n, -1) * gate) @ w["o"].T, S.transpose(1, 2).contiguous()


def _exact_ssm(case, w, x, c, row, tables, storage):
    s, n = _sizes(case), x.shape[0]
    H, V, N, G = s["heads"], s["vdim"], s["state"], s["groups"]
    inner, bc = H * V, G * N
    z = x @ w["in"].T
    gate, dt = z[:, :inner], torch.nn.functional.softplus(z[:, 2 * inner + 2 * bc :] + w["dt_bias"])
    z = _silu(_convolve(z[:, inner : 2 * inner + 2 * bc], storage.states[1][row].double(), w["conv"]) + w["conv.b"])
    v = z[:, :inner].view(n, H, V)
    B = z[:, inner : inner + bc].view(n, G, N).repeat_interleave(H // G, dim=1)
    C = z[:, inner + bc :].view(n, G, N).repeat_interleave(H // G, dim=1)
    g = torch.exp(-torch.exp(w["A_log"]) * dt)
    S = storage.states[0][row].double()  # [H, V, N]
    outs = []
    for t in range(n):
        S = S * g[t][:, None, None] + (dt[t][:, None] * v[t])[:, :, None] * B[t][:, None]
        outs.append(torch.bmm(S, C[t][:, :, None])[..., 0])
    y = ((torch.stack(outs) + w["D"][:, None] * v).reshape(n, inner) * _silu(gate)).view(n, G, inner // G)
    y = (y * torch.rsqrt(y.square().mean(-1, keepdim=True) + EPS)).view(n, inner) * w["norm"]
    return y @ w["o"].T, S


def _exact_moe(case, w, x):
    s = _sizes(case)
    logits = x @ w["router"].T + w["router.b"]
    top, ids = torch.topk(logits, s["top"], dim=-1)
    weights = torch.softmax(top, dim=-1)
    out = torch.zeros_like(x)
    for e in range(s["experts"]):
        token, place = (ids == e).nonzero(as_tuple=True)
        if token.numel():
            a = (x[token] @ w[f"e{e}.gate"].T).clamp(max=s["limit"])
            b = (x[token] @ w[f"e{e}.up"].T).clamp(-s["limit"], s["limit"])
            rows = (a * torch.sigmoid(s["alpha"] * a) * (b + s["shift"])) @ w[f"e{e}.down"].T
            out.index_add_(0, token, rows * weights[token, place][:, None])
    return out


def _exact_serve(case, seed):
    width, heads = case["width"], case["width"] // 128
    kv = width // 512
    model, _ = build_model(_dense_config(case), dtype=case["dtype"], device="meta")  # for the tensors' names
    w = _weights(model.tensor_specs(), DTYPES[case["dtype"]], seed)

    def norm(h, name):
        return h * torch.rsqrt(h.square().mean(-1, keepdim=True) + EPS) * w[name].double()

    rows = []
    for prompt, told in _dialogue(case, seed):
        tokens = torch.tensor(prompt + told, device=DEVICE)
        n = len(tokens)
        at = torch.arange(n, device=DEVICE)
        h = w["model.embed_tokens.weight"][tokens].double()
        for layer in range(8):
            p = f"model.layers.{layer}."
            m = {name: w[p + name].double() for name in ("self_attn.q_proj.weight", "self_attn.k_proj.weight", "self_attn.v_proj.weight", "self_attn.o_proj.weight",
                                                         "mlp.gate_proj.weight", "mlp.up_proj.weight", "mlp.down_proj.weight")}
            y = norm(h, p + "input_layernorm.weight")
            q = _turn((y @ m["self_attn.q_proj.weight"].T).view(n, heads, 128), at, 128)
            k = _turn((y @ m["self_attn.k_proj.weight"].T).view(n, kv, 128), at, 128)
            v = (y @ m["self_attn.v_proj.weight"].T).view(n, kv, 128)
            h = h + _attend(q, k, v, 0, 128 ** -0.5).reshape(n, -1) @ m["self_attn.o_proj.weight"].T
            y = norm(h, p + "post_attention_layernorm.weight")
            h = h + (_silu(y @ m["mlp.gate_proj.weight"].T) * (y @ m["mlp.up_proj.weight"].T)) @ m["mlp.down_proj.weight"].T
        wanted = norm(h[len(prompt) - 1 :], "model.norm.weight")
        rows.append(wanted @ w["lm_head.weight"].double().T)
    return torch.stack(rows, dim=1)
