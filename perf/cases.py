"""Performance cases: the calls that users of this library make, over the sizes they make them at.

Four kinds of pass, each through the public Python entry points:

* `generate` - one conversation turn on a session: `prefill_argmax` of the prompt, then one
  `decode_argmax` call per token (or `decode`, which also hands out the logits, where a sampler or a
  repetition penalty needs them). The continuation is given instead of fed back, so that one near-tie
  of two logits changes one token and not all that follow;
* `prompt`   - scoring a prompt: `prefill`, logits of the last position out;
* `batch`    - serving several sequences: `step` calls that decode every slot once;
* `linear`   - one fused dequantise-and-multiply product, `ops.linear`.

Models are the Qwen3 shapes of `dyninfer_b200.synth`; the large ones are cut to a few layers, each of
which does the full model's work. Weights are seeded synthetic checkpoints written on first use.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

from dyninfer_b200 import checkpoint, ops, synth
from dyninfer_b200.runtime import ModelLoader, SessionConfig

WEIGHT_SEED = 20242
MIXED = {"attn_v": "gguf.q4_1", "ffn_down": "gguf.q8_0"}
# name -> (shape, encoding per linear, encoding of the tied embedding / lm_head)
MODELS = {
    "0.6b-q4_0": (synth.QWEN3_0_6B, dict.fromkeys(synth.linear_shapes(synth.QWEN3_0_6B), "gguf.q4_0"), "gguf.q6_k"),
    "0.6b-mlx": (synth.QWEN3_0_6B, dict.fromkeys(synth.linear_shapes(synth.QWEN3_0_6B), "mlx.affine.u4"), "plain.bf16"),
    "8b-mixed": (dict(synth.QWEN3_8B, layers=8),
                 {**dict.fromkeys(synth.linear_shapes(synth.QWEN3_8B), "gguf.q4_0"), **MIXED}, "gguf.q6_k"),
    "32b-q4_0": (dict(synth.QWEN3_32B, layers=2), dict.fromkeys(synth.linear_shapes(synth.QWEN3_32B), "gguf.q4_0"),
                 "gguf.q6_k"),
}
# stored bytes per weight; MLX: 4 bits plus a bf16 scale and bias per 64 weights
BYTES = {"gguf.q4_0": 18 / 32, "gguf.q4_1": 20 / 32, "gguf.q8_0": 34 / 32, "gguf.q6_k": 210 / 256,
         "gguf.q4_k": 144 / 256, "gguf.q5_k": 176 / 256, "gguf.iq4_xs": 136 / 256, "mlx.affine.u4": 0.5 + 4 / 64,
         "plain.bf16": 2.0}
KV_BYTES = {"f32": 4, "bf16": 2, "f16": 2}


def listed():
    return [
        # the headline: a short chat turn, one call per token
        {"name": "chat 0.6b q4_0", "kind": "generate", "model": "0.6b-q4_0", "kv": "bf16", "prompt": 16, "new": 128,
         "logits": False},
        # a longer turn on an MLX checkpoint
        {"name": "chat 0.6b mlx", "kind": "generate", "model": "0.6b-mlx", "kv": "bf16", "prompt": 512, "new": 256,
         "logits": False},
        # sampling on the host: every step hands out its logits
        {"name": "sample 8b mixed", "kind": "generate", "model": "8b-mixed", "kv": "f16", "prompt": 100, "new": 60,
         "logits": True},
        # time to first token of a short question, the loader's default cache type
        {"name": "prompt 0.6b 37", "kind": "prompt", "model": "0.6b-q4_0", "kv": "f32", "prompt": 37},
        # a document that fills the default session, the loader's default cache type
        {"name": "prompt 0.6b 2048", "kind": "prompt", "model": "0.6b-q4_0", "kv": "f32", "prompt": 2048},
        # a document on a larger model; the length does not end on a chunk
        {"name": "prompt 8b 1531", "kind": "prompt", "model": "8b-mixed", "kv": "bf16", "prompt": 1531},
        # serving a few users
        {"name": "serve 0.6b mlx x8", "kind": "batch", "model": "0.6b-mlx", "kv": "bf16", "slots": 8, "context": 512,
         "steps": 32},
        # serving many
        {"name": "serve 0.6b q4_0 x64", "kind": "batch", "model": "0.6b-q4_0", "kv": "bf16", "slots": 64,
         "context": 200, "steps": 16},
        # serving a few users with long contexts on a larger model
        {"name": "serve 8b mixed x8", "kind": "batch", "model": "8b-mixed", "kv": "bf16", "slots": 8, "context": 2048,
         "steps": 16},
        # a single product of a small model's layer: launches and host work count
        {"name": "linear q4_0 3072x1024 m1", "kind": "linear", "enc": "gguf.q4_0", "n": 3072, "k": 1024, "m": 1,
         "x": "f32"},
        # the lm_head of one token
        {"name": "linear q6_k lm_head m1", "kind": "linear", "enc": "gguf.q6_k", "n": 151936, "k": 1024, "m": 1,
         "x": "bf16"},
        # a prefill chunk through a feed-forward matrix
        {"name": "linear q8_0 12288x4096 m512", "kind": "linear", "enc": "gguf.q8_0", "n": 12288, "k": 4096, "m": 512,
         "x": "bf16"},
    ]


def _log(rng, low, high):
    """A whole number between the two, spread evenly over the logarithm."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choice(["generate", "prompt", "batch", "linear", "linear"])
    if kind == "linear":
        enc = rng.choice(["gguf.q4_0", "gguf.q4_1", "gguf.q8_0", "gguf.q6_k", "gguf.q4_k", "mlx.affine.u4"])
        k = 256 * _log(rng, 2, 100)
        n = _log(rng, 512, min(151936, (160 << 20) // k))
        m = _log(rng, 1, min(2048, 12288 * 4096 * 2048 // (n * k)))
        return {"kind": kind, "enc": enc, "n": n, "k": k, "m": m, "x": rng.choice(["f32", "bf16"])}
    model = rng.choice(sorted(MODELS))
    kv = rng.choice(["f32", "bf16", "f16"])
    if kind == "generate":
        logits = rng.random() < 0.3
        return {"kind": kind, "model": model, "kv": kv, "prompt": _log(rng, 4, 1024),
                "new": _log(rng, 8, 62) if logits else _log(rng, 100, 200), "logits": logits}
    if kind == "prompt":
        return {"kind": kind, "model": model, "kv": kv, "prompt": _log(rng, 8, 2048 if kv == "f32" else 4096)}
    slots = _log(rng, 2, 64)
    return {"kind": kind, "model": model, "kv": "bf16" if kv == "f32" else kv, "slots": slots,
            "context": _log(rng, 32, min(2048, 16384 // slots)), "steps": max(16, -(-200 // slots))}


def _checkpoint(model):
    """Path of the model's seeded checkpoint, written by whoever needs it first."""
    shape, encodings, embed = MODELS[model]
    folder = os.path.join(tempfile.gettempdir(), f"dyninfer_perf_{os.getuid()}")
    os.makedirs(folder, exist_ok=True)
    mlx = "mlx.affine.u4" in encodings.values()
    path = os.path.join(folder, model + ("" if mlx else ".gguf"))
    if not os.path.exists(path):
        part = f"{path}.{os.getpid()}"
        if mlx:
            synth.write_qwen3_mlx(part, shape, seed=WEIGHT_SEED)
        else:
            synth.write_qwen3_gguf(part, shape, seed=WEIGHT_SEED, encodings=encodings, embd=embed, repeat_layers=True)
            _signs(part)
        try:
            os.rename(part, path)
        except OSError:      # another process was first
            pass
    return path


def _signs(path):
    """Scales of either sign, as quantisers write them. With positive ones only, every weight has the same small
    negative mean, which through the layers drowns all else: any prompt would give the same token."""
    rng = np.random.default_rng(WEIGHT_SEED)
    scales = {"gguf.q4_0": (18, [1]), "gguf.q4_1": (20, [1, 3]), "gguf.q6_k": (210, range(192, 208))}
    for p in checkpoint.open_catalog(path).parameters.values():
        if p.encoding not in scales:
            continue
        size, at = scales[p.encoding]
        c = p.components[0]
        blocks = np.memmap(path, np.uint8, "r+", c.offset, (c.length // size, size))
        for column in at if p.encoding == "gguf.q6_k" else [at]:    # Q6_K has a scale of its own per 16 weights
            minus = rng.integers(0, 2, size=c.length // size, dtype=np.uint8)
            if p.encoding == "gguf.q6_k":
                blocks[:, column] = (blocks[:, column] ^ -minus) + minus
            else:
                blocks[:, column] ^= (minus << 7)[:, None]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    if case["kind"] == "linear":
        n, k, m = case["n"], case["k"], case["m"]
        t = synth.random_weight(case["enc"], n, k, seed)
        s.weight = ops.DeviceWeight(case["enc"], n, k, t["packed"], t["scales"], t["biases"]) \
            if case["enc"] == "mlx.affine.u4" else ops.DeviceWeight(case["enc"], n, k, t["data"])
        g = torch.Generator("cuda").manual_seed(seed)
        s.x = torch.randn(m, k, generator=g, device="cuda")
        if case["x"] == "bf16":
            s.x = s.x.to(torch.bfloat16)
        return s
    rng = np.random.default_rng(seed)
    vocab = MODELS[case["model"]][0]["vocab"]

    def ids(count):
        return rng.integers(0, vocab, size=count).tolist()

    slots, length = case.get("slots", 1), case.get("prompt", case.get("context"))
    limit = max(2048, length + case.get("new", case.get("steps", 0)))
    model = ModelLoader().load(_checkpoint(case["model"]), max_kv=limit, kv_dtype=case["kv"])
    config = SessionConfig(max_sequence_length=limit, batch_size=slots)
    if case["kind"] == "batch":
        # the sequences are in the cache already: a pass decodes on from there
        s.session = model.create_batched_session(config)
        for slot in range(slots):
            s.session.prefill_slot(slot, ids(length))
        s.feed = [dict(enumerate(ids(slots))) for _ in range(case["steps"])]
        return s
    s.session = model.create_session(config)
    s.prompt = ids(length)
    s.follow = ids(case.get("new", 0))
    return s


def run(state):
    case = state.case
    if case["kind"] == "linear":
        return ops.linear(state.weight, state.x)
    session = state.session
    if case["kind"] == "prompt":
        return session.prefill(state.prompt).values
    if case["kind"] == "batch":
        session.positions = [case["context"]] * case["slots"]
        made = [session.step(tokens) for tokens in state.feed]
        return np.array([[step[slot] for slot in range(case["slots"])] for step in made])
    if case["logits"]:
        first = session.prefill(state.prompt).values
        return [first] + [session.decode(token).values for token in state.follow]
    first = session.prefill_argmax(state.prompt)
    made = [session.decode_argmax(token) for token in state.follow[:-1]]
    return {"tokens": np.array([first] + made), "logits": session.decode(state.follow[-1]).values}


def _weights(case):
    """(bytes, count) of the weights that one step reads: the layers' linears, and the lm_head."""
    shape, encodings, embed = MODELS[case["model"]]
    sizes = {slot: n * k * shape["layers"] for slot, (n, k) in synth.linear_shapes(shape).items()}
    head = shape["vocab"] * shape["hidden"]
    return (sum(BYTES[encodings[s]] * v for s, v in sizes.items()), sum(sizes.values()), BYTES[embed] * head, head)


def work(case):
    if case["kind"] == "linear":
        n, k, m = case["n"], case["k"], case["m"]
        return {"bytes": BYTES[case["enc"]] * n * k + m * k * (4 if case["x"] == "f32" else 2) + 4 * m * n,
                "flops": 2 * m * n * k}
    shape = MODELS[case["model"]][0]
    layer_bytes, layer_count, head_bytes, head_count = _weights(case)
    token_kv = 2 * shape["layers"] * shape["kv_heads"] * shape["head_dim"] * KV_BYTES[case["kv"]]
    score = 4 * shape["layers"] * shape["heads"] * shape["head_dim"]    # flops per (query, key) pair
    if case["kind"] == "batch":
        steps, slots = case["steps"], case["slots"]
        keys = slots * sum(case["context"] + i + 1 for i in range(steps))
        return {"bytes": steps * (layer_bytes + head_bytes) + token_kv * (keys + steps * slots),
                "flops": 2 * steps * slots * (layer_count + head_count) + score * keys}
    p, new = case["prompt"], case.get("new", 0)
    keys = sum(p + i + 1 for i in range(new))
    return {"bytes": (1 + new) * (layer_bytes + head_bytes) + token_kv * (p + keys + new)
            + 4 * shape["vocab"] * ((1 + new) if case.get("logits") else 1),
            "flops": 2 * (p + new) * layer_count + 2 * (1 + new) * head_count + score * (p * (p + 1) // 2 + keys)}


def tolerance(case):
    if case["kind"] == "linear":
        # up to four rows: exact products, 32-bit sums; more rows: operands rounded to 11 bits
        return {"rel": 1e-5 if case["m"] <= 4 else 1e-3}
    # prompt and batched products round their operands to 11 bits, a 2-byte cache its entries to 8 or 11,
    # through every layer; a token differs where two logits tie within that
    return {"rel": 5e-3, "differ": 0.01}
