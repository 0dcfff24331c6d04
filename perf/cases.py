"""Performance cases: the work a user of this package has it do, through its public entry points.

``listed()`` names the cases that are always timed, ``draw(rng)`` gives further ones of the same ranges.
A case is a dict of plain values; ``prepare`` turns it into what a user's program holds before the call,
``run`` makes one pass, ``work`` states what the pass cannot do without, ``tolerance`` how close another
correct implementation has to come.

Kinds of pass:

``decode``       one step of a host-driven loop: ``DecoderKernel.decode``, logits come back
``generate``     a few greedy steps sampled on the device: ``DecoderKernel.decode_steps``
``host_step``    one greedy step from and to pinned host memory, synchronised: ``DecoderKernel.step_from_host``
``ragged``       one step of a batch whose sequences have different lengths: ``DecoderKernel.decode_ragged``
``prefill``      a stateless prompt pass: ``DecoderKernel.prefill``
``kv_attention`` the decode attention op alone: ``torch.ops.megabake.kv_attention``
``attention``    the prompt attention op alone: ``torch.ops.megabake.attention``

Decode passes start from a cache that already holds ``context`` positions of every sequence.  A pass puts
the valid lengths (and, where the call advances them, ids and positions) back to the start of the step first,
as a program does that tries another continuation of the same prefix, so that every pass does the same work.

Weights are random: unit-variance embeddings, N(0, 0.02) projections, the projections that write to the
residual stream divided by sqrt(2 * layers).  The residual stream is then led by the token's own embedding, as
it is in trained models, and two correct bf16 evaluations of 24 to 32 layers stay close enough to be compared;
with N(0, 0.02) throughout they differ by several per cent.  The output head holds the embedding rows moved by
one, so the greedy continuation is certain and does not hang on the last bit of two logits.
"""

from __future__ import annotations

import dataclasses
import math

import torch

from megabake_b200 import ops  # noqa: F401  registers torch.ops.megabake
from megabake_b200.runtime import DecoderKernel
from megabake_b200.synth import CONFIGS, DecoderConfig, weight_names

DEVICE = "cuda"
HEAD_SHAPES = ((9, 3, 64), (14, 2, 64), (32, 32, 64), (32, 8, 128))  # (query heads, key/value heads, head size) of CONFIGS


def listed() -> list[dict]:
    return [
        # the smallest model, one user, a short reply generated without the host: launches and hand-offs only
        dict(name="generate-135m-b1", kind="generate", model="smollm-135m", batch=1, context=48, capacity=128, steps=16),
        # a small model with biases and grouped heads, one user, the host picks every token
        dict(name="decode-0.5b-b1", kind="decode", model="qwen2-0.5b", batch=1, context=99, capacity=128),
        # the headline shape: one user served step by step from the host, half a cache filled
        dict(name="host-step-1.7b-b1", kind="host_step", model="smollm-1.7b", batch=1, context=1024, capacity=2048),
        # a few users at an odd context
        dict(name="decode-1.7b-b3", kind="decode", model="smollm-1.7b", batch=3, context=777, capacity=1024),
        # one stream of the data-parallel sweep: eight sequences from a 512-token prefix, device-side sampler
        dict(name="generate-1.7b-b8", kind="generate", model="smollm-1.7b", batch=8, context=512, capacity=768, steps=4),
        # an ordinary serving batch
        dict(name="decode-1.7b-b16", kind="decode", model="smollm-1.7b", batch=16, context=1024, capacity=2048),
        # continuous batching: six sequences, each at a place of its own
        dict(name="ragged-1.7b-b6", kind="ragged", model="smollm-1.7b", batch=6, context=1500, capacity=2048),
        # the largest: a full batch on the largest shape, untied head, long contexts
        dict(name="decode-8b-b32", kind="decode", model="llama3-8b", batch=32, context=2048, capacity=2304),
        # prompts: a short one that fills its bucket, a long one that does not
        dict(name="prefill-1.7b-64", kind="prefill", model="smollm-1.7b", batch=1, sequence=64, masked=False),
        dict(name="prefill-1.7b-500", kind="prefill", model="smollm-1.7b", batch=1, sequence=500, masked=False),
        # the two ops as a captured or eager model calls them
        dict(name="kv-attention-b16", kind="kv_attention", heads=32, kv_heads=32, head_dim=64, batch=16, context=1024, capacity=2048),
        dict(name="attention-512", kind="attention", heads=32, kv_heads=32, head_dim=64, batch=1, sequence=512, masked=True),
    ]


def _log_uniform(rng, low: int, high: int) -> int:
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng) -> dict:
    kind = rng.choice(("generate", "decode", "decode", "decode", "host_step", "ragged", "prefill", "prefill", "kv_attention",
                       "attention"))
    if kind == "prefill":
        batch = rng.choice((1, 1, 1, 2, 3, 4))
        return dict(kind=kind, model=rng.choice(("smollm-135m", "qwen2-0.5b", "smollm-1.7b", "smollm-1.7b")), batch=batch,
                    sequence=_log_uniform(rng, 8, 512 // batch), masked=rng.random() < 0.25)
    if kind == "attention":
        heads, kv_heads, head_dim = rng.choice(HEAD_SHAPES)
        batch = rng.choice((1, 1, 2, 4))
        return dict(kind=kind, heads=heads, kv_heads=kv_heads, head_dim=head_dim, batch=batch,
                    sequence=_log_uniform(rng, 16, 1024 // batch), masked=rng.random() < 0.75)
    batch, context = _log_uniform(rng, 1, 32), _log_uniform(rng, 16, 2048)
    if kind in ("generate", "host_step"):
        batch = _log_uniform(rng, 1, 16)
    capacity = context + rng.randint(16, 256)
    if kind == "kv_attention":
        heads, kv_heads, head_dim = rng.choice(HEAD_SHAPES)
        return dict(kind=kind, heads=heads, kv_heads=kv_heads, head_dim=head_dim, batch=batch, context=context, capacity=capacity)
    models = ("smollm-135m", "qwen2-0.5b", "smollm-1.7b", "smollm-1.7b") + (() if kind == "generate" else ("llama3-8b",))
    case = dict(kind=kind, model=rng.choice(models), batch=batch, context=context, capacity=capacity)
    if kind == "generate":
        case["steps"] = rng.randint(2, 16)
        while case["steps"] > 1 and work(case)["bytes"] > 20e9:  # no more than the largest listed case
            case["steps"] -= 1
    return case


# ----------------------------------------------------------------------------- inputs
def _normal(generator, shape, std: float = 1.0) -> torch.Tensor:
    return torch.empty(shape, dtype=torch.bfloat16, device=DEVICE).normal_(0.0, std, generator=generator)


def _weights(config: DecoderConfig, generator) -> dict[str, torch.Tensor]:
    weights = {}
    residual_std = 0.02 / math.sqrt(2 * config.layers)
    for name, shape, kind in weight_names(config):
        if kind == "ones":
            weights[name] = 1.0 + _normal(generator, shape, 0.1)
        elif name == "model.embed_tokens.weight":
            weights[name] = _normal(generator, shape)
        elif name.endswith(("o_proj.weight", "down_proj.weight")):
            weights[name] = _normal(generator, shape, residual_std)
        elif name != "lm_head.weight":
            weights[name] = _normal(generator, shape, 0.02)
    weights["lm_head.weight"] = weights["model.embed_tokens.weight"].roll(1, 0)
    return weights


def _lengths(case) -> list[int]:
    """Filled positions of every sequence: ``context`` for all, or spread evenly below it for ``ragged``."""
    if case["kind"] != "ragged":
        return [case["context"]] * case["batch"]
    return [max(1, case["context"] * (row + 1) // case["batch"] - 3 * row) for row in range(case["batch"])]


def prepare(case: dict, seed: int) -> dict:
    generator = torch.Generator(device=DEVICE).manual_seed(seed)
    state = dict(case=case)
    batch = case["batch"]
    if case["kind"] in ("kv_attention", "attention"):
        heads, kv_heads, dim = case["heads"], case["kv_heads"], case["head_dim"]
        length = 1 if case["kind"] == "kv_attention" else case["sequence"]
        state["query"] = _normal(generator, (batch, length, heads, dim))
        state["key"] = _normal(generator, (batch, length, kv_heads, dim))
        state["value"] = _normal(generator, (batch, length, kv_heads, dim))
        if case["kind"] == "kv_attention":
            state["cache"] = _normal(generator, (2, batch, case["capacity"], kv_heads, dim))
            state["length"] = torch.full((1,), case["context"], dtype=torch.int32, device=DEVICE)
        else:
            state["mask"] = _causal(batch, length) if case["masked"] else None
        return state

    config = CONFIGS[case["model"]]
    config = dataclasses.replace(config, tied=False)
    weights = _weights(config, generator)
    state["config"] = config
    if case["kind"] == "prefill":
        sequence = case["sequence"]
        state["kernel"] = DecoderKernel(config, weights, max_tokens=batch * sequence, max_positions=max(sequence, 16), device=DEVICE)
        state["ids"] = torch.randint(0, config.vocab, (batch, sequence), device=DEVICE, generator=generator)
        state["positions"] = torch.arange(sequence, device=DEVICE).expand(batch, sequence).contiguous()
        state["mask"] = _causal(batch, sequence) if case["masked"] else None
        return state

    capacity = case["capacity"]
    state["kernel"] = DecoderKernel(config, weights, max_tokens=batch, max_positions=capacity, device=DEVICE)
    state["caches"] = _normal(generator, (2, config.layers, batch, capacity, config.kv_heads, config.head_dim))
    lengths = torch.tensor(_lengths(case), dtype=torch.int32, device=DEVICE)
    per_layer = batch if case["kind"] == "ragged" else 1
    state["start_lengths"] = lengths[:per_layer].expand(config.layers, per_layer).contiguous()
    state["lengths"] = state["start_lengths"].clone()
    state["start_io"] = torch.stack((torch.randint(0, config.vocab, (batch, 1), device=DEVICE, generator=generator),
                                     lengths.to(torch.int64).view(batch, 1)))
    state["io"] = state["start_io"].clone()  # ids, positions
    state["kv"] = ([*state["caches"][0]], [*state["caches"][1]], [*state["lengths"]])
    if case["kind"] == "host_step":
        state["host"] = [tensor.cpu().pin_memory() for tensor in state["io"]]
        state["host_tokens"] = torch.zeros((batch, 1), dtype=torch.int64).pin_memory()
    return state


def _causal(batch: int, length: int) -> torch.Tensor:
    """The additive mask transformers builds for a prompt: the most negative bf16 above the diagonal."""
    mask = torch.full((length, length), torch.finfo(torch.bfloat16).min, dtype=torch.bfloat16, device=DEVICE).triu(1)
    return mask.expand(batch, 1, length, length).contiguous()


# ----------------------------------------------------------------------------- one pass
def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "attention":
        return torch.ops.megabake.attention(state["query"], state["key"], state["value"], state["mask"], case["head_dim"] ** -0.5)
    if kind == "kv_attention":
        state["length"].fill_(case["context"])
        out = torch.ops.megabake.kv_attention(state["query"], state["key"], state["value"], state["cache"][0], state["cache"][1],
                                              state["length"])
        return out, state["cache"], state["length"]
    kernel = state["kernel"]
    if kind == "prefill":
        return kernel.prefill(state["ids"], state["positions"], state["mask"])
    state["lengths"].copy_(state["start_lengths"])
    ids, positions = state["io"]
    if kind == "generate":
        state["io"].copy_(state["start_io"])
        tokens, logits = kernel.decode_steps(ids, positions, *state["kv"], steps=case["steps"], return_logits=True)
        return tokens, logits, state["io"], state["caches"], state["lengths"]
    if kind == "host_step":
        tokens = kernel.step_from_host(*state["host"], *state["kv"], state["host_tokens"])
        return tokens, state["caches"], state["lengths"]
    step = kernel.decode_ragged if kind == "ragged" else kernel.decode
    logits = step(ids, positions, *state["kv"])
    return logits, state["caches"], state["lengths"]


# ----------------------------------------------------------------------------- what a pass cannot do without
def work(case: dict) -> dict:
    batch = case["batch"]
    if case["kind"] == "attention":
        sequence, dim = case["sequence"], case["head_dim"]
        pairs = batch * sequence * (sequence + 1) // 2 if case["masked"] else batch * sequence * sequence
        rows = batch * sequence * dim * (2 * case["heads"] + 2 * case["kv_heads"])
        return dict(bytes=2 * rows + (2 * batch * sequence * sequence if case["masked"] else 0), flops=4 * pairs * case["heads"] * dim)
    if case["kind"] == "kv_attention":
        keys, dim = case["context"] + 1, case["head_dim"]
        rows = 2 * case["kv_heads"] * (keys + 1) + 2 * case["heads"]
        return dict(bytes=2 * batch * rows * dim, flops=4 * batch * keys * case["heads"] * dim)
    config = CONFIGS[case["model"]]
    parameters = config.streamed_parameters()
    if case["kind"] == "prefill":
        sequence = case["sequence"]
        tokens = batch * sequence
        pairs = batch * sequence * (sequence + 1) // 2
        return dict(bytes=2 * parameters + 2 * tokens * (config.hidden + config.vocab),
                    flops=2 * parameters * tokens + 4 * pairs * config.q_size * config.layers)
    keys = steps = 0
    for step in range(case.get("steps", 1)):
        keys += sum(length + step + 1 for length in _lengths(case))
        steps += 1
    kv_row = 2 * config.layers * config.kv_size * 2
    return dict(bytes=2 * parameters * steps + kv_row * keys + 2 * steps * batch * (config.hidden + config.vocab),
                flops=2 * parameters * batch * steps + 4 * keys * config.q_size * config.layers)


def tolerance(case: dict) -> dict:
    # bf16 results of one op: one rounding of the output, and probabilities rounded to bf16 before they are used.
    if case["kind"] in ("attention", "kv_attention"):
        return dict(rel=5e-3)
    # 24 to 32 layers of bf16 tensors, each rounded where the layer before differed in its last bits: the two decode
    # engines and eager PyTorch on one GPU are 0.3 % (135M), 0.5 % (0.5B) and 1.0-1.2 % (1.7B) apart on these weights.
    # Sampled tokens are whole numbers and stay the same (the continuation is certain, see above).
    return dict(rel=2e-2)
