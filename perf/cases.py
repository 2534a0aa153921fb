"""Timed cases of the engine: what a serving program has it do, from the smallest calls to the largest.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare(case, seed)`` makes what a
program holds before the call (an engine with seeded random weights, requests with cached tokens, prompts), ``run(state)``
is one pass through the public entry points and returns its outputs, ``work(case)`` says what the pass cannot do without,
``exact(case, seed)`` computes the same outputs in 64 bits with plain torch, and ``tolerance(case)`` says how far two
correct implementations may be apart.

Kinds of cases:

* ``decode``: one decode step (``StepRunner.decode_sampled``) of ``batch`` requests that hold ``context`` cached tokens
  each, greedy, as the scheduler issues it: the step is launched, then the tokens of the step before are read.  Before every
  pass the requests are put back to the end of their context, so that any number of passes does the same work.  Outputs: the
  logits and what the step wrote into the pages (the states of mixers that keep one go on from pass to pass).
* ``prefill``: the prompts of ``prompts`` requests, ``tokens`` in all, in one step (``StepRunner.step``), the logits of every
  prompt's last token, and everything the step left in the cache.
* ``mixed``: one step of continuous batching (``StepRunner.step_sampled``): a portion of a prompt behind ``cached`` tokens of
  it, beside one token each of ``batch`` decoding requests of different lengths.
* ``generate``: ``Engine.generate`` from prompts to tokens, prompts cut into portions of ``portion`` tokens a step.
* ``sample``: ``Sampler.sample`` on ``rows`` rows of logits, every row with options of its own.

Models: the Qwen3-8B shape (the benchmark's headline) with a quarter of its 36 layers (through all of them the bfloat16 roundings
of two correct implementations drift apart by 0.03 of the logits, through nine by half of that), the Qwen3-0.6B shape (where launches and small products count), a
tiny Qwen3 in float32 (latency of the host and of the launches alone), and the two designs without routed experts among the
hybrids (Sorulix, Fumolorn) at the sizes of the benchmark's comparisons.  Designs with routed experts are left out: two
correct bfloat16 implementations may send a token to different experts, after which their outputs cannot be compared.
"""

from __future__ import annotations

import math
import random
from types import SimpleNamespace

import torch

PAGE_SIZE = 16
QWEN3 = {
    "architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "hidden_act": "silu", "attention_bias": False,
    "attention_dropout": 0.0, "rms_norm_eps": 1e-6, "rope_theta": 1000000.0, "head_dim": 128, "max_position_embeddings": 8192,
    "vocab_size": 151936, "bos_token_id": 151643, "eos_token_id": 151645,
}
DELTA_UNIT_EPS, GLU_ALPHA, DISTANCE_BASE = 1e-6, 1.702, 8.0     # constants of the Sorulix design
NORMALISER_EPS = 1e-6                                           # of the Fumolorn design


# --------------------------------------------------------------------------------------------------------------- models
def _hybrid_sizes(size: str) -> tuple[int, int, int, int, int, int]:
    """(width, feed-forward, heads, key/value heads, head size, vocabulary); four layers."""

    return {"2k": (2048, 8192, 16, 4, 128, 32000), "4k": (4096, 12288, 32, 8, 128, 32000)}[size]


def _sorulix(size: str) -> dict:
    width, ff, heads, kv_heads, d, vocab = _hybrid_sizes(size)
    parallel = {"type": "parallel", "mixer": {
        "left": {"heads": heads, "kv_heads": kv_heads, "dim": d, "vdim": d, "scale": d ** -0.5, "softcap": 50.0,
                 "q_temp": {"coef": 0.3, "every": 64}},
        "right": {"heads": heads, "dim": d, "vdim": d, "decay": [1.0 - 2.0 ** (-5 - 3 * h / heads) for h in range(heads)]}},
        "mlp": {"kind": "dense", "ff": ff, "limit": 7.0}}
    delta = {"type": "channel_delta", "mixer": {"heads": heads, "kv_heads": heads, "dim": d, "vdim": d, "conv": 4},
             "mlp": {"kind": "dense", "ff": ff, "limit": 7.0}}
    return {"architecture": "Sorulix", "vocab": vocab, "width": width, "norm": {"eps": 1e-6}, "torch_dtype": "bfloat16",
            "layers": [parallel, delta] * 2}


def _fumolorn(size: str) -> dict:
    width, ff, heads, _, d, vocab = _hybrid_sizes(size)
    latent = {"heads": heads, "dim": d, "rot_dim": d // 2, "vdim": d, "kv_rank": 4 * d, "q_rank": width // 2, "scale": (d + d // 2) ** -0.5,
              "rot": {"base": 10000.0, "dims": d // 2, "scaling": {"factor": 4.0, "original": 4096, "fast": 24.0, "slow": 2.0}}}
    mlp = {"kind": "dense", "ff": ff}
    layers = [{"type": "gla", "mixer": {"heads": heads, "dim": d, "vdim": d, "tau": 8.0}, "mlp": mlp},
              {"type": "latent_attention", "mixer": latent, "mlp": mlp},
              {"type": "mlstm", "mixer": {"heads": heads, "dim": d, "vdim": d, "gate_cap": 15.0}, "mlp": mlp},
              {"type": "latent_attention", "mixer": latent, "mlp": mlp}]
    return {"architecture": "Fumolorn", "vocab": vocab, "width": width, "norm": {"eps": 1e-6}, "torch_dtype": "bfloat16",
            "residual_mult": 0.5, "logit_softcap": 25.0, "layers": layers,
            "embedding": {"scale": width ** 0.5, "bigram": {"buckets": 65521, "mul_prev": 131, "mul_cur": 17}}}


def _config(case: dict) -> dict:
    """The ``config.json`` of the case's model."""

    model, dtype = case["model"], case["dtype"]
    if model == "qwen3-8b":
        return {**QWEN3, "hidden_size": 4096, "intermediate_size": 12288, "num_hidden_layers": 9, "num_attention_heads": 32,
                "num_key_value_heads": 8, "tie_word_embeddings": False, "torch_dtype": dtype}
    if model == "qwen3-0.6b":
        return {**QWEN3, "hidden_size": 1024, "intermediate_size": 3072, "num_hidden_layers": 28, "num_attention_heads": 16,
                "num_key_value_heads": 8, "tie_word_embeddings": True, "torch_dtype": dtype}
    if model == "qwen3-tiny":
        return {**QWEN3, "hidden_size": 96, "intermediate_size": 272, "num_hidden_layers": 3, "num_attention_heads": 6,
                "num_key_value_heads": 1, "head_dim": 32, "vocab_size": 503, "max_position_embeddings": 512, "rms_norm_eps": 1e-5,
                "tie_word_embeddings": False, "torch_dtype": dtype, "bos_token_id": 0, "eos_token_id": [501, 502]}
    family, size = model.split("-")
    return {"sorulix": _sorulix, "fumolorn": _fumolorn}[family](size)


def _vocab(config: dict) -> int:
    return config.get("vocab_size", config.get("vocab"))


# ---------------------------------------------------------------------------------------------------------------- cases
def listed() -> list[dict]:
    return [
        # A handful of short prompts through the Python entry point of a tiny float32 model: the latency of host and launches.
        {"name": "generate-tiny-fp32", "kind": "generate", "model": "qwen3-tiny", "dtype": "float32", "prompts": 5, "longest": 70,
         "new_tokens": 12, "portion": 13},
        # One user's chat with a small model: every launch and every small product counts.
        {"name": "decode-0.6b-b1-509", "kind": "decode", "model": "qwen3-0.6b", "dtype": "bfloat16", "batch": 1, "context": 509},
        # The benchmark's headline: eight requests with 2,048 cached tokens each.
        {"name": "decode-8b-b8-2048", "kind": "decode", "model": "qwen3-8b", "dtype": "bfloat16", "batch": 8, "context": 2048},
        # A full server: 64 requests of about a thousand tokens.
        {"name": "decode-8b-b64-1011", "kind": "decode", "model": "qwen3-8b", "dtype": "bfloat16", "batch": 64, "context": 1011},
        # The benchmark's prompt, in one step.
        {"name": "prefill-8b-2048", "kind": "prefill", "model": "qwen3-8b", "dtype": "bfloat16", "prompts": 1, "tokens": 2048},
        # Continuous batching: a portion of a long prompt beside running requests; an odd number of rows in every product.
        {"name": "mixed-8b-381-24", "kind": "mixed", "model": "qwen3-8b", "dtype": "bfloat16", "batch": 24, "portion": 381, "cached": 640,
         "longest": 1500},
        # The 32-bit run type, which logits are verified in: a prompt of the length the reference reports.
        {"name": "prefill-0.6b-fp32-509", "kind": "prefill", "model": "qwen3-0.6b", "dtype": "float32", "prompts": 1, "tokens": 509},
        # Drawing tokens for 32 users with options of their own from a large vocabulary.
        {"name": "sample-32", "kind": "sample", "rows": 32, "vocab": 151936},
        # A hybrid's prompt: attention with rules beside linear attention, and the delta rule.
        {"name": "prefill-sorulix-4k-2048", "kind": "prefill", "model": "sorulix-4k", "dtype": "bfloat16", "prompts": 1, "tokens": 2048},
        # A hybrid's decode step at a middling batch.
        {"name": "decode-sorulix-2k-b32-1024", "kind": "decode", "model": "sorulix-2k", "dtype": "bfloat16", "batch": 32, "context": 1024},
        # Three prompts of different lengths in one step: latent attention, matrix memories, gated linear attention.
        {"name": "prefill-fumolorn-4k-3x1733", "kind": "prefill", "model": "fumolorn-4k", "dtype": "bfloat16", "prompts": 3, "tokens": 1733},
        {"name": "decode-fumolorn-4k-b8-2048", "kind": "decode", "model": "fumolorn-4k", "dtype": "bfloat16", "batch": 8, "context": 2048},
    ]


def _between(rng: random.Random, low: int, high: int) -> int:
    """A whole number of [low, high], spread evenly over its logarithm."""

    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(("decode", "decode", "decode", "prefill", "prefill", "prefill", "mixed", "generate", "sample"))
    if kind == "generate":
        prompts = rng.randint(1, 8)
        return {"kind": kind, "model": "qwen3-tiny", "dtype": "float32", "prompts": prompts, "longest": _between(rng, 8, 96),
                "new_tokens": rng.randint(4, 16), "portion": _between(rng, 8, 64)}
    if kind == "sample":
        return {"kind": kind, "rows": _between(rng, 1, 64), "vocab": _between(rng, 500, 151936)}
    if kind == "mixed":
        return {"kind": kind, "model": rng.choice(("qwen3-0.6b", "qwen3-8b")), "dtype": "bfloat16", "batch": _between(rng, 1, 28),
                "portion": _between(rng, 16, 1024), "cached": rng.randint(0, 1024), "longest": _between(rng, 64, 2048)}
    model = rng.choice(("qwen3-0.6b", "qwen3-8b", "sorulix-2k", "sorulix-4k", "fumolorn-2k", "fumolorn-4k"))
    dtype = "float32" if model == "qwen3-0.6b" and rng.random() < 0.3 else "bfloat16"
    if kind == "decode":
        most = 64 if model.startswith("qwen3") else 32
        batch = _between(rng, 1, most)
        return {"kind": kind, "model": model, "dtype": dtype, "batch": batch, "context": _between(rng, 64, min(4096, 65536 // batch))}
    prompts = rng.randint(1, 4)
    return {"kind": kind, "model": model, "dtype": dtype, "prompts": prompts,
            "tokens": _between(rng, 16 * prompts, 1024 if dtype == "float32" else 2048)}


def _generator(seed: int) -> torch.Generator:
    return torch.Generator().manual_seed(0x5EED0000 + seed)


def _cut(total: int, parts: int, rng: random.Random) -> list[int]:
    """``total`` as ``parts`` lengths, every one at least one token and of a size of its own."""

    weights = [rng.uniform(0.5, 1.5) for _ in range(parts)]
    lengths = [max(1, int(total * w / sum(weights))) for w in weights]
    lengths[0] += total - sum(lengths)
    return lengths


def _prompts(case: dict, seed: int) -> SimpleNamespace:
    """Everything about the case's requests that is drawn from the seed: token ids, lengths, pending tokens."""

    vocab, generator, rng = _vocab(_config(case)), _generator(seed), random.Random(0)     # lengths belong to the case, not to the seed

    def ids(n: int) -> list[int]:
        return torch.randint(0, vocab, (n,), generator=generator).tolist()

    kind = case["kind"]
    if kind == "prefill":
        return SimpleNamespace(prompts=[ids(n) for n in _cut(case["tokens"], case["prompts"], rng)])
    if kind == "generate":
        lengths = [rng.randint(1, case["longest"]) for _ in range(case["prompts"] - 1)] + [case["longest"]]
        return SimpleNamespace(prompts=[ids(n) for n in lengths])
    if kind == "decode":
        return SimpleNamespace(prompts=[ids(case["context"]) for _ in range(case["batch"])], pending=ids(case["batch"]))
    lengths = [rng.randint(max(1, case["longest"] // 4), case["longest"]) for _ in range(case["batch"])]
    return SimpleNamespace(prompts=[ids(n) for n in lengths], pending=ids(case["batch"]), cached=ids(case["cached"]), portion=ids(case["portion"]))


# -------------------------------------------------------------------------------------------------------------- prepare
def _engine(case: dict, seed: int, *, requests: int, lengths: list[int], **options):
    from llm_runtime_study_b200.engine.engine import Engine

    pages = sum(-(-n // PAGE_SIZE) for n in lengths)
    longest = min(-(-max(lengths) // 1024) * 1024, _config(case).get("max_position_embeddings", 1 << 30))
    return Engine.from_random_weights(_config(case), seed=seed, device="cuda:0", dtype=case["dtype"], max_seq_len=longest,
                                      max_batch_size=requests, page_size=PAGE_SIZE, max_cache_tokens=pages * PAGE_SIZE, **options)


def _feed(runner, request, tokens: list[int]) -> None:
    """Run ``tokens`` of a request into the cache, in portions."""

    from llm_runtime_study_b200.engine.step import StepEntry

    for at in range(0, len(tokens), 2048):
        runner.step([StepEntry(request, tokens[at : at + 2048])])


def _written(manager, request, first: int, last: int) -> dict:
    """Views of the pages' slots that hold positions ``first`` to ``last`` of a request (whole pages, if there are several)."""

    out = {}
    for g, pool in enumerate(manager.groups):
        size = pool.page_size
        pages = request.tables[g][first // size : last // size + 1]
        assert pages == list(range(pages[0], pages[0] + len(pages)))
        for name, tensor in pool.tensors.items():
            kept = tensor[:, pages[0] : pages[-1] + 1]
            out[f"g{g}.{name}"] = kept.select(-2, last % size) if first == last else kept
    return out


def prepare(case: dict, seed: int):
    from llm_runtime_study_b200.cache.slots import SlotRecord
    from llm_runtime_study_b200.sampling import Sampler, SamplingConfig

    kind = case["kind"]
    if kind == "sample":
        generator = torch.Generator(device="cuda").manual_seed(seed)
        logits = 2.5 * torch.randn((case["rows"], case["vocab"]), generator=generator, device="cuda")
        options = (SamplingConfig(), SamplingConfig(temperature=0.7), SamplingConfig(temperature=0.8, top_k=min(50, case["vocab"])),
                   SamplingConfig(temperature=0.9, top_p=0.9), SamplingConfig(temperature=1.0, top_k=min(200, case["vocab"]), top_p=0.95))
        rows = [(options[i % len(options)], 1000 * seed + i, 7 + i) for i in range(case["rows"])]
        return SimpleNamespace(kind=kind, logits=logits, rows=rows, sampler=Sampler(torch.device("cuda", 0), max_rows=case["rows"]))
    made = _prompts(case, seed)
    if kind == "generate":
        lengths = [len(p) + case["new_tokens"] for p in made.prompts]
        engine = _engine(case, seed, requests=len(lengths), lengths=[512] * len(lengths), max_tokens_per_step=case["portion"])
        state = SimpleNamespace(kind=kind, engine=engine, prompts=made.prompts, new_tokens=case["new_tokens"])
        list(engine.generate([[1, 2, 3]] * len(lengths), max_new_tokens=2))
        return state
    if kind == "prefill":
        lengths = [len(p) for p in made.prompts]
        engine = _engine(case, seed, requests=len(lengths), lengths=lengths)
        manager = engine.cache_manager
        kept = {f"g{g}.{name}": t for g, pool in enumerate(manager.groups) for name, t in pool.tensors.items()}
        kept.update({f"s{i}": t[: len(lengths)] for i, t in enumerate(manager.state_arrays.values())})
        return SimpleNamespace(kind=kind, engine=engine, runner=engine.runner, manager=manager, prompts=made.prompts, kept=kept)
    # requests with cached tokens and a pending token in their slot records
    mixed = kind == "mixed"
    lengths = [len(p) + 1 for p in made.prompts] + ([case["cached"] + case["portion"]] if mixed else [])
    engine = _engine(case, seed, requests=len(lengths), lengths=lengths)
    runner, manager = engine.runner, engine.cache_manager
    requests = [manager.admit() for _ in lengths]
    for request, n in zip(requests, lengths):
        manager.grow(request, n)
    for request, prompt in zip(requests, made.prompts + ([made.cached] if mixed else [])):
        _feed(runner, request, prompt)
    state = SimpleNamespace(kind=kind, engine=engine, runner=runner, manager=manager, sampler=engine._sampler, requests=requests,
                            starts=[r.length for r in requests], before=None, made=made, greedy=SlotRecord(position=0))
    if mixed:
        state.kept = {f"r{i}": _written(manager, r, s, s) for i, (r, s) in enumerate(zip(requests[:-1], state.starts))}
        state.kept["portion"] = _written(manager, requests[-1], case["cached"], case["cached"] + case["portion"] - 1)
        return state
    for request, token, start in zip(requests, made.pending, state.starts):
        manager.slots.note(request.slot, SlotRecord(position=start, last_token=token))
    state.records = torch.from_numpy(manager.slots.mirror.copy()).to(manager.device)
    states = {key: array.clone() for key, array in manager.state_arrays.items()}
    _decode(state)                              # the program has decoded before: the step is captured
    for key, array in states.items():
        manager.state_arrays[key].copy_(array)
    n, at = len(requests), case["context"]
    state.kept = {}
    for g, pool in enumerate(manager.groups):   # every request holds as many pages, one behind the other
        size = pool.page_size
        step = at // size + 1
        assert [r.tables[g][-1] for r in requests] == [i * step + step - 1 for i in range(n)]
        for name, tensor in pool.tensors.items():
            state.kept[f"g{g}.{name}"] = tensor[:, step - 1 : n * step : step].select(-2, at % size)
    state.kept.update({f"s{i}": t[:n] for i, t in enumerate(manager.state_arrays.values())})
    return state


# ------------------------------------------------------------------------------------------------------------------ run
def _decode(state):
    """One decode step of all requests from the end of their contexts; the tokens of the step before are read behind its launch."""

    for request, start in zip(state.requests, state.starts):
        if request.length > start:
            state.manager.rollback(request, start)
    state.manager.slots.records.copy_(state.records)
    handle, before = state.runner.decode_sampled(state.requests, state.sampler), state.before
    state.before = handle
    if before is not None:
        before.tokens()
    return state.runner.last_logits


def run(state):
    if state.kind == "sample":
        return {"tokens": torch.tensor(state.sampler.sample(state.logits, state.rows))}
    if state.kind == "generate":
        tokens = [[] for _ in state.prompts]
        for index, event in state.engine.generate(state.prompts, max_new_tokens=state.new_tokens):
            tokens[index].append(-1 if event.token_id is None else event.token_id)
        padded = [row + [-1] * (state.new_tokens - len(row)) for row in tokens]
        return {"tokens": torch.tensor(padded), "last_logits": state.engine.runner.last_logits}
    if state.kind == "decode":
        return {"logits": _decode(state), **state.kept}
    from llm_runtime_study_b200.engine.step import StepEntry

    if state.kind == "prefill":
        requests = [state.manager.admit() for _ in state.prompts]
        logits = state.runner.step([StepEntry(r, p, [len(p) - 1]) for r, p in zip(requests, state.prompts)])
        for request in reversed(requests):
            state.manager.release(request)
        return {"logits": logits, **state.kept}
    for request, start in zip(state.requests, state.starts):
        if request.length > start:
            state.manager.rollback(request, start)
    entries = [StepEntry(r, [t], [0], state.greedy) for r, t in zip(state.requests, state.made.pending)]
    entries.append(StepEntry(state.requests[-1], state.made.portion, [len(state.made.portion) - 1], state.greedy))
    handle, before = state.runner.step_sampled(entries, state.sampler), state.before
    state.before = handle
    if before is not None:
        before.tokens()
    return {"logits": state.runner.last_logits, **state.kept}


# ----------------------------------------------------------------------------------------------------------------- work
def _schema(config: dict) -> dict:
    from llm_runtime_study_b200.config import architecture_for
    from llm_runtime_study_b200.models.description import tensor_schema

    arch = architecture_for(config)
    return {n: s for n, s in tensor_schema(arch.describe(arch.config_from_dict(config))).items() if not s.optional}


def _is_table(name: str) -> bool:
    return "embed" in name or name == "bigram"


def work(case: dict) -> dict:
    """Bytes: every weight once (one row a token of the embedding tables), the cache rows that are read and written, states in
    and out, logits out.  Operations: two per weight and row, and those of attention scores, weighted sums and state updates."""

    if case["kind"] == "sample":
        return {"bytes": 4.0 * case["rows"] * (case["vocab"] + 1), "flops": 0.0}
    config, made = _config(case), _prompts(case, 0)
    vocab, size = _vocab(config), 4 if case["dtype"] == "float32" else 2
    if case["kind"] == "prefill":
        spans, wanted = [(0, len(p)) for p in made.prompts], len(made.prompts)
    elif case["kind"] == "generate":
        spans, wanted = [(0, len(p) + case["new_tokens"] - 1) for p in made.prompts], case["new_tokens"] * len(made.prompts)
    else:
        spans, wanted = [(len(p), 1) for p in made.prompts], len(made.prompts)
        if case["kind"] == "mixed":
            spans, wanted = spans + [(case["cached"], case["portion"])], wanted + 1
    tokens = sum(n for _, n in spans)
    pairs = sum(n * start + n * (n + 1) / 2 for start, n in spans)      # (query, visible key)
    schema = _schema(config)
    head = next((s for n, s in schema.items() if n in ("head", "lm_head.weight")), None)
    head_size = vocab * (config.get("hidden_size") or config.get("width"))
    matrices = sum(math.prod(s.shape) for n, s in schema.items() if len(s.shape) > 1 and not _is_table(n)) - (head_size if head else 0)
    steps = case["new_tokens"] if case["kind"] == "generate" else 1     # a generated token needs the weights again
    flops = 2.0 * tokens * matrices + 2.0 * wanted * head_size
    moved = float(steps * size * (matrices + head_size) + 4 * wanted * vocab)
    if config.get("model_type") == "qwen3":
        layers, d = config["num_hidden_layers"], config["head_dim"]
        flops += 4.0 * layers * config["num_attention_heads"] * d * pairs
        moved += 2.0 * size * layers * config["num_key_value_heads"] * d * sum(start + n for start, n in spans)
        return {"bytes": moved, "flops": flops}
    for layer in config["layers"]:
        m, kind = layer["mixer"], layer["type"]
        if kind == "parallel":
            left = m["left"]
            flops += 4.0 * left["heads"] * left["dim"] * pairs
            moved += 2.0 * size * left["kv_heads"] * left["dim"] * sum(start + n for start, n in spans)
            m = m["right"]
        if kind == "latent_attention":
            flops += 2.0 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]) * pairs
            moved += size * (m["kv_rank"] + m["rot_dim"]) * sum(start + n for start, n in spans)
            continue
        state = m["heads"] * m["dim"] * m["vdim"]
        flops += (6.0 if kind == "channel_delta" else 4.0) * state * tokens
        moved += 4.0 * state * sum(1 + (start > 0) for start, _ in spans)
    return {"bytes": moved, "flops": flops}


def tolerance(case: dict):
    """bfloat16: other kernels for the same products, norms and attention were seen to move logits by 0.004 to 0.016 and single cache
    entries near zero by 0.5 of the root mean square.  float32: the logits are 2e-6 from their values in 64 bits."""

    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 2e-3, "differ": 0.0}
    return {"rel": 0.03, "max": 0.9}


# ---------------------------------------------------------------------------------------------------------- in 64 bits
def _weights(config: dict, seed: int) -> dict:
    """The model's seeded random weights as they are stored, on the GPU."""

    from llm_runtime_study_b200.weights.random_init import random_tensor

    dtype = {"float32": torch.float32, "bfloat16": torch.bfloat16}[config["torch_dtype"]]
    return {n: random_tensor(n, s, seed, dtype=dtype, device="cuda") for n, s in _schema(config).items()}


class _Wide:
    """The weights under a prefix, widened to 64 bits when they are asked for."""

    def __init__(self, weights: dict, prefix: str = "") -> None:
        self.weights, self.prefix = weights, prefix

    def __getitem__(self, name: str) -> torch.Tensor:
        return self.weights[self.prefix + name].double()

    def __contains__(self, name: str) -> bool:
        return self.prefix + name in self.weights

    def sub(self, prefix: str) -> "_Wide":
        return _Wide(self.weights, f"{self.prefix}{prefix}.")

    def map(self, x: torch.Tensor, name: str) -> torch.Tensor:
        return x @ self[name].T


def _unit(x: torch.Tensor, eps: float) -> torch.Tensor:
    return x / torch.sqrt(x.square().mean(dim=-1, keepdim=True) + eps)


def _silu(x: torch.Tensor) -> torch.Tensor:
    return x * torch.sigmoid(x)


def _attend(q, k, v, scores, sink=None) -> torch.Tensor:
    """q ``[T, H, d]``, k, v ``[T, G, .]``; ``scores(s, h)`` turns a head's products into scores; ``sink[h]``: the score of a
    key without a value."""

    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    hidden = torch.ones((T, T), dtype=torch.bool, device=q.device).triu(1)
    out = torch.empty((T, H, v.shape[2]), dtype=q.dtype, device=q.device)
    for h in range(H):
        g = h // (H // G)
        s = scores(q[:, h] @ k[:, g].T, h).masked_fill(hidden, -math.inf)
        top = s.max(dim=-1, keepdim=True).values
        if sink is not None:
            top = torch.maximum(top, sink[h])
        e = torch.exp(s - top)
        total = e.sum(dim=-1, keepdim=True)
        out[:, h] = (e / (total if sink is None else total + torch.exp(sink[h] - top))) @ v[:, g]
    return out


def _qwen3_layers(w: _Wide, config: dict, sequences: list[list[int]]):
    """The rows behind the last layer and, per layer, the keys and values, all sequences side by side."""

    H, G, d, eps = config["num_attention_heads"], config["num_key_value_heads"], config["head_dim"], config["rms_norm_eps"]
    lengths = [len(s) for s in sequences]
    ids = torch.tensor([t for s in sequences for t in s], device="cuda")
    x = w.weights["model.embed_tokens.weight"][ids].double()
    dims = torch.arange(0, d, 2, dtype=torch.float32, device="cuda")
    positions = torch.cat([torch.arange(n, device="cuda") for n in lengths])
    angles = (positions.to(torch.float32)[:, None] * (1.0 / (config["rope_theta"] ** (dims / d)))).double()
    cos, sin = angles.cos().repeat(1, 2)[:, None], angles.sin().repeat(1, 2)[:, None]

    def rotate(a: torch.Tensor) -> torch.Tensor:
        return a * cos + torch.cat((-a[..., d // 2 :], a[..., : d // 2]), dim=-1) * sin

    keys, values = [], []
    for i in range(config["num_hidden_layers"]):
        p = w.sub(f"model.layers.{i}")
        a = p.sub("self_attn")
        h = _unit(x, eps) * p["input_layernorm.weight"]
        q = rotate(_unit(a.map(h, "q_proj.weight").view(-1, H, d), eps) * a["q_norm.weight"])
        k = rotate(_unit(a.map(h, "k_proj.weight").view(-1, G, d), eps) * a["k_norm.weight"])
        v = a.map(h, "v_proj.weight").view(-1, G, d)
        o = torch.cat([_attend(qs, ks, vs, lambda s, _: s * d ** -0.5) for qs, ks, vs in zip(q.split(lengths), k.split(lengths), v.split(lengths))])
        x = x + a.map(o.reshape(-1, H * d), "o_proj.weight")
        h, m = _unit(x, eps) * p["post_attention_layernorm.weight"], p.sub("mlp")
        x = x + m.map(_silu(m.map(h, "gate_proj.weight")) * m.map(h, "up_proj.weight"), "down_proj.weight")
        keys.append(k)
        values.append(v)
    return x, {"g0.keys": keys, "g0.values": values}


def _qwen3_head(w: _Wide, config: dict, x: torch.Tensor) -> torch.Tensor:
    x = _unit(x, config["rms_norm_eps"]) * w["model.norm.weight"]
    return w.map(x, "lm_head.weight" if "lm_head.weight" in w else "model.embed_tokens.weight")


def _scan(q, k, u, lengths, *, decay=None, gate=None, beta=None, gates=None) -> torch.Tensor:
    """``S <- D S + k u^T``, ``o = S^T q`` token after token, the sequences side by side; ``decay`` ``[H]`` or ``gate`` ``[N, H, d]``;
    ``beta`` ``[N, H]``: the delta rule; ``gates``: (log input gate, log forget gate) ``[N, H]`` of a matrix memory, whose read-outs are
    divided by their normaliser."""

    device, starts = q.device, torch.tensor([sum(lengths[:i]) for i in range(len(lengths))], device=q.device)
    H, d, dv = q.shape[1], q.shape[2], u.shape[2]
    out = torch.empty((q.shape[0], H, dv), dtype=q.dtype, device=device)
    S = torch.zeros((len(lengths), H, d, dv), dtype=q.dtype, device=device)
    n = torch.zeros((len(lengths), H, d), dtype=q.dtype, device=device)
    m = torch.zeros((len(lengths), H), dtype=q.dtype, device=device)
    order = torch.tensor(sorted(range(len(lengths)), key=lambda i: -lengths[i]), device=device)      # longest first: those still going are in front
    starts = starts[order]
    ordered = sorted(lengths, reverse=True)
    for t in range(ordered[0]):
        going = sum(length > t for length in ordered)
        at = starts[:going] + t
        kt, qt, ut, St = k[at], q[at], u[at], S[:going]
        if gates is not None:
            log_i, log_f = gates[0][at], gates[1][at]
            top = torch.maximum(log_f + m[:going], log_i)
            forget, take = torch.exp(log_f + m[:going] - top), torch.exp(log_i - top)
            m[:going] = top
            St.mul_(forget[..., None, None])
            n[:going] = forget[..., None] * n[:going] + take[..., None] * kt
            ut = take[..., None] * ut
        else:
            St.mul_(decay[None, :, None, None] if decay is not None else gate[at][..., None])
        if beta is not None:
            ut = beta[at][..., None] * (ut - (St * kt[..., None]).sum(dim=2))
        St.addcmul_(kt[..., None], ut[..., None, :])
        o = (St * qt[..., None]).sum(dim=2)
        if gates is not None:
            o = o / (torch.maximum((n[:going] * qt).sum(-1).abs(), torch.exp(-m[:going])) + NORMALISER_EPS)[..., None]
        out[at] = o
    return out


def _sorulix_layers(w: _Wide, config: dict, sequences: list[list[int]]):
    eps = config["norm"]["eps"]
    lengths = [len(s) for s in sequences]
    x = w.weights["embed"][torch.tensor([t for s in sequences for t in s], device="cuda")].double()
    positions = torch.cat([torch.arange(n, device="cuda") for n in lengths])
    keys, values = [], []

    def convolved(a: torch.Tensor, taps: torch.Tensor) -> torch.Tensor:
        parts = []
        for rows in a.split(lengths):
            padded = torch.cat((rows.new_zeros(taps.shape[1] - 1, rows.shape[1]), rows))
            parts.append(sum(padded[j : j + rows.shape[0]] * taps[:, j] for j in range(taps.shape[1])))
        return _silu(torch.cat(parts))

    def unit_heads(a: torch.Tensor) -> torch.Tensor:
        return a / torch.sqrt(a.square().sum(-1, keepdim=True) + DELTA_UNIT_EPS)

    for i, layer in enumerate(config["layers"]):
        p = w.sub(f"l{i}")
        h, mix = _unit(x, eps) * (1.0 + p["norm1"]), p.sub("mix")
        if layer["type"] == "parallel":
            c, a = layer["mixer"]["left"], mix.sub("left")
            H, G, d, cap = c["heads"], c["kv_heads"], c["dim"], c["softcap"]
            q = _unit(a.map(h, "q"), eps) * a["q.norm"]
            steps = torch.div(positions + 1, c["q_temp"]["every"], rounding_mode="floor").double()
            q = (q * (1.0 + c["q_temp"]["coef"] * torch.log(steps + 1.0))[:, None]).view(-1, H, d)
            k, v = (_unit(a.map(h, "k"), eps) * a["k.norm"]).view(-1, G, d), a.map(h, "v").view(-1, G, d)
            parts = []
            for qs, ks, vs in zip(q.split(lengths), k.split(lengths), v.split(lengths)):
                at = torch.arange(qs.shape[0], device="cuda", dtype=torch.float64)
                distance = at[:, None] - at[None, :]

                def scores(s, head):
                    return cap * torch.tanh(s * c["scale"] / cap) - 2.0 ** (-DISTANCE_BASE * (head + 1) / H) * distance

                parts.append(_attend(qs, ks, vs, scores, torch.zeros(H, dtype=torch.float64, device="cuda")))
            left = a.map(torch.cat(parts).reshape(-1, H * d), "o")
            keys.append(k)
            values.append(v)
            c, a = layer["mixer"]["right"], mix.sub("right")
            H, d = c["heads"], c["dim"]
            q, k, v = (_silu(a.map(h, name)).view(-1, H, d) for name in ("q", "k", "v"))
            o = _scan(q, k, v, lengths, decay=torch.tensor(c["decay"], dtype=torch.float64, device="cuda")).reshape(-1, H * d)
            right = a.map(_unit(o, eps) * a["norm"] * torch.sigmoid(a.map(h, "g")), "o")
            x = x + 0.5 * (_unit(left, eps) * mix["left.out"] + _unit(right, eps) * mix["right.out"])
        else:
            c = layer["mixer"]
            H, d = c["heads"], c["dim"]
            q, k, v = (convolved(mix.map(h, name), mix[f"{name}.conv"]).view(-1, H, d) for name in ("q", "k", "v"))
            rate = torch.nn.functional.softplus(mix.map(mix.map(h, "a1"), "a2") + mix["dt_bias"]).view(-1, H, d)
            o = _scan(unit_heads(q) * d ** -0.5, unit_heads(k), v, lengths, gate=torch.exp(-torch.exp(mix["A_log"])[:, None] * rate),
                      beta=torch.sigmoid(mix.map(h, "b")))
            o = _unit(o, eps) * mix["norm"] * torch.sigmoid(mix.map(mix.map(h, "g1"), "g2")).view(-1, H, d)
            x = x + mix.map(o.reshape(-1, H * d), "o")
        h, m, limit = _unit(x, eps) * (1.0 + p["norm2"]), p.sub("mlp"), layer["mlp"]["limit"]
        g = torch.clamp(m.map(h, "gate") + m["gate.b"], max=limit)
        u = torch.clamp(m.map(h, "up") + m["up.b"], min=-limit, max=limit)
        x = x + m.map(g * torch.sigmoid(GLU_ALPHA * g) * (u + 1.0), "down") + m["down.b"]
    return x, {"g0.keys": keys, "g0.values": values}


def _sorulix_head(w: _Wide, config: dict, x: torch.Tensor) -> torch.Tensor:
    return w.map(_unit(x, config["norm"]["eps"]) * (1.0 + w["final.norm"]), "embed")


def _yarn(rot: dict) -> tuple[torch.Tensor, float]:
    """Frequencies of the pairs and the factor on cosine and sine."""

    dims, base, s = rot["dims"], rot["base"], rot["scaling"]

    def index(turns: float) -> float:
        return dims * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))

    low, high = max(math.floor(index(s["fast"])), 0), min(math.ceil(index(s["slow"])), dims - 1)
    at = torch.arange(dims // 2, dtype=torch.float64, device="cuda")
    plain, ramp = base ** (-2.0 * at / dims), ((at - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
    return plain / s["factor"] * ramp + plain * (1.0 - ramp), 0.1 * math.log(s["factor"]) + 1.0


def _fumolorn_layers(w: _Wide, config: dict, sequences: list[list[int]]):
    eps, e = config["norm"]["eps"], config["embedding"]
    lengths = [len(s) for s in sequences]
    ids, bigram = torch.tensor([t for s in sequences for t in s], device="cuda"), e["bigram"]
    pairs = [bigram["buckets"] if t == 0 else (s[t - 1] * bigram["mul_prev"] + token * bigram["mul_cur"]) % bigram["buckets"]
             for s in sequences for t, token in enumerate(s)]
    x = w.weights["embed"][ids].double() * e["scale"] + w.weights["bigram"][torch.tensor(pairs, device="cuda")].double()
    x = _unit(x, eps) * w["embed.norm"]
    positions = torch.cat([torch.arange(n, device="cuda") for n in lengths]).double()
    kept = []

    def log_sigmoid(z):
        return -torch.nn.functional.softplus(-z)

    for i, layer in enumerate(config["layers"]):
        p, c = w.sub(f"l{i}"), layer["mixer"]
        a, H, d, dv = p.sub("mix"), c["heads"], c["dim"], c["vdim"]
        if layer["type"] == "latent_attention":
            freq, factor = _yarn(c["rot"])
            angle = positions[:, None] * freq
            cos, sin = factor * angle.cos(), factor * angle.sin()

            def rotate(z, cos=cos, sin=sin):
                z = z.unflatten(-1, (-1, 2))
                shape = (z.shape[0],) + (1,) * (z.dim() - 3) + (z.shape[-2],)
                cc, ss = cos.view(shape), sin.view(shape)
                return torch.stack((z[..., 0] * cc - z[..., 1] * ss, z[..., 1] * cc + z[..., 0] * ss), dim=-1).flatten(-2)

            rank, scale = c["kv_rank"], c["scale"]
            q = a.map(_unit(a.map(x, "dq"), eps) * a["dq.norm"], "uq").view(-1, H, d + c["rot_dim"])
            q = torch.cat((q[..., :d], rotate(q[..., d:])), dim=-1)
            down = a.map(x, "dkv")
            latent, turned = _unit(down[:, :rank], eps) * a["dkv.norm"], rotate(down[:, rank:])
            k = torch.cat((a.map(latent, "uk").view(-1, H, d), turned[:, None].expand(-1, H, -1)), dim=-1)
            v = a.map(latent, "uv").view(-1, H, dv)
            o = torch.cat([_attend(qs, ks, vs, lambda s, _: s * scale, a["sink"])
                           for qs, ks, vs in zip(q.split(lengths), k.split(lengths), v.split(lengths))])
            out = a.map((o * torch.sigmoid(a.map(x, "g"))[..., None]).reshape(-1, H * dv), "o")
            kept.append(torch.cat((latent, turned), dim=-1))
        else:
            q, k, v = a.map(x, "q").view(-1, H, d) * d ** -0.5, a.map(x, "k").view(-1, H, d), a.map(x, "v").view(-1, H, dv)
            if layer["type"] == "gla":
                alpha = torch.exp(log_sigmoid(a.map(a.map(x, "a1"), "a2") + a["a2.b"]) / c["tau"]).view(-1, H, d)
                o = (_unit(_scan(q, k, v, lengths, gate=alpha), eps) * a["norm"]).reshape(-1, H * dv) * _silu(a.map(x, "g"))
            else:
                cap = c["gate_cap"]
                log_i = cap * torch.tanh((a.map(x, "i") + a["i.b"]) / cap)
                log_f = log_sigmoid(cap * torch.tanh((a.map(x, "f") + a["f.b"]) / cap))
                o = _unit(_scan(q, k, v, lengths, gates=(log_i, log_f)), eps).reshape(-1, H * dv) * a["norm"] * torch.sigmoid(a.map(x, "g"))
            out = a.map(o, "o")
        x = x + config["residual_mult"] * _unit(out, eps) * p["norm1"]
        m = p.sub("mlp")
        out = m.map(torch.nn.functional.gelu(m.map(x, "gate"), approximate="tanh") * m.map(x, "up"), "down")
        x = x + config["residual_mult"] * _unit(out, eps) * p["norm2"]
    return x, {"g0.latent": kept}


def _fumolorn_head(w: _Wide, config: dict, x: torch.Tensor) -> torch.Tensor:
    cap = config["logit_softcap"]
    return cap * torch.tanh(w.map(_unit(x, config["norm"]["eps"]) * w["final.norm"], "head") / cap)


def _plain(config: dict):
    family = "qwen3" if config.get("model_type") == "qwen3" else config["architecture"].lower()
    return {"qwen3": (_qwen3_layers, _qwen3_head), "sorulix": (_sorulix_layers, _sorulix_head),
            "fumolorn": (_fumolorn_layers, _fumolorn_head)}[family]


def exact(case: dict, seed: int):
    """Logits and cache rows of the first pass in 64 bits; ``None`` where that would take too long.  Pages of prefilled prompts
    and the mixers' states are left to the logits, which read them."""

    kind = case["kind"]
    if kind == "sample":
        return None
    config, made = _config(case), _prompts(case, seed)
    layers, head = _plain(config)
    if kind == "generate":
        sequences = [list(p) for p in made.prompts]
        w = _Wide(_weights(config, seed))
        for _ in range(case["new_tokens"]):
            x, _kept = layers(w, config, sequences)
            last = torch.tensor([sum(len(s) for s in sequences[: i + 1]) - 1 for i in range(len(sequences))], device="cuda")
            logits = head(w, config, x[last])
            for sequence, token in zip(sequences, logits.argmax(dim=-1).tolist()):
                sequence.append(token)
        if any(t in config["eos_token_id"] for p, s in zip(made.prompts, sequences) for t in s[len(p) :]):
            return None                     # some request ends early
        # the last prompt is the longest and is fed last: the last step is its alone, or holds more rows than this
        return {"last_logits": logits[-1:]}
    if kind == "decode":
        sequences = [p + [t] for p, t in zip(made.prompts, made.pending)]
    elif kind == "prefill":
        sequences = made.prompts
    else:
        sequences = [p + [t] for p, t in zip(made.prompts, made.pending)] + [made.cached + made.portion]
    schema = _schema(config)
    total = sum(math.prod(s.shape) for n, s in schema.items() if not _is_table(n))
    if 2.0 * total * sum(len(s) for s in sequences) > 3.5e14:          # about ten seconds of 64-bit products
        return None
    w = _Wide(_weights(config, seed))
    x, kept = layers(w, config, sequences)
    last = torch.tensor([sum(len(s) for s in sequences[: i + 1]) - 1 for i in range(len(sequences))], device="cuda")
    out = {"logits": head(w, config, x[last])}
    if kind == "decode":
        out.update({name: torch.stack([rows[last] for rows in per_layer]) for name, per_layer in kept.items() if name.startswith("g0")})
    return out
