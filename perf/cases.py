"""The work that users of this package have it do, as cases that can be timed and compared.

A case is a dict of plain values; `prepare` puts in place what a program holds before the call (checkpoint, engine or
op table with its buffers, inputs drawn from a seed), `run` is one pass through the public entry points. Shapes are
those of this repository's benchmark configurations and tests, and of the ranges around them:

  forward      `Pi0Inference.forward`: one control decision, images + state + noise in, action chunk out. Camera views,
               prompt length, chunk, Euler steps and episodes per replay vary with the robot and the server.
  prefill      `pipeline.vision_encoder` + `pipeline.transformer_encoder` through the op table: the prefix KV cache alone.
  decode       `pipeline.transformer_decoder` through the op table, on a prefix KV cache that is already there.
  decoder_ffn  two call sites of the op table on the action expert's few rows (gated FFN, down projection).
  encoder_ffn  the same two call sites of the prefix encoder.

One checkpoint, drawn from a fixed seed, serves every case of a process, and an engine serves every state of its
configuration: that is how a program uses them, new inputs arrive at an engine that exists. Inputs follow the seed.
"""
from __future__ import annotations

import functools
import math

import torch

from flash_vla_b200 import Pi0Inference, op_table, random_checkpoint
from flash_vla_b200.hardware.nvidia.b200.pi0 import pipeline
from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import wrappers
from flash_vla_b200.hardware.nvidia.b200.pi0.buffers import allocate_static_buffers
from flash_vla_b200.models.pi0 import spec
from flash_vla_b200.runtime.cuda import ScratchPool

bf16 = torch.bfloat16
VOCAB_ROWS = 16384           # rows of the embedding table that prompts draw their ids from
MAX_PREFIX_ROWS = 8 * 768    # prefix tokens of all episodes of one replay
MAX_DECODER_ROWS = 8 * 51    # action-expert rows of all episodes of one replay


def _forward(name, views, prompt=0, table=False, chunk=50, steps=10, episodes=1):
    case = {"kind": "forward", "views": views, "prompt": prompt, "table": table, "chunk": chunk, "steps": steps,
            "episodes": episodes}
    return dict(case, name=name) if name else case


def listed():
    return [
        # the smallest calls: a program with its own orchestration that calls the action expert's FFN through the table
        {"name": "decoder_ffn_51", "kind": "decoder_ffn", "tokens": 51},
        # the isolated prefix-encoder FFN of the GEMM sweep
        {"name": "encoder_ffn_768", "kind": "encoder_ffn", "tokens": 768},
        # one diffusion step on a given prefix cache: 51 rows, 819 keys
        {"name": "decode_one_step", "kind": "decode", "views": 3, "prompt": 0, "chunk": 50, "steps": 1},
        # the prefix cache alone, with a prompt that makes the row count ragged
        {"name": "prefill_prompt48", "kind": "prefill", "views": 3, "prompt": 48},
        # a one-camera robot with a short chunk, half the Euler steps and an odd prompt
        _forward("forward_1view_short", 1, prompt=17, chunk=10, steps=5),
        # one camera, full chunk
        _forward("forward_1view", 1),
        # the published shape: three cameras, empty prompt
        _forward("forward_3views", 3),
        # the same with a prompt of 256 tokens, looked up inside the pass
        _forward("forward_prompt256", 3, prompt=256, table=True),
        # a longer chunk and an odd prompt: 65 decoder rows, 817 prefix rows
        _forward("forward_chunk64", 3, prompt=49, chunk=64),
        # servers that batch episodes: two, four (the throughput configuration) and eight in one replay
        _forward("forward_2episodes", 3, episodes=2),
        _forward("forward_4episodes", 3, prompt=48, episodes=4),
        _forward("forward_8episodes", 3, episodes=8),
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["forward"] * 7 + ["decode", "prefill", "decoder_ffn", "encoder_ffn"])
    if kind == "decoder_ffn":
        return {"kind": kind, "tokens": _log_int(rng, 2, 65)}
    if kind == "encoder_ffn":
        return {"kind": kind, "tokens": _log_int(rng, 256, 1280)}
    views = rng.choice((1, 3, 3, 4))
    prompt = rng.choice((0, 1)) * _log_int(rng, 4, 256)
    if kind == "prefill":
        return {"kind": kind, "views": views, "prompt": prompt}
    chunk = rng.choice((50, _log_int(rng, 8, 64)))
    if kind == "decode":
        return {"kind": kind, "views": views, "prompt": prompt, "chunk": chunk, "steps": rng.randint(1, 10)}
    steps = rng.choice((10, rng.randint(4, 10)))
    most = min(8, MAX_PREFIX_ROWS // (views * spec.VISION_TOKENS + prompt), MAX_DECODER_ROWS // (chunk + 1))
    episodes = rng.choice((1, _log_int(rng, 1, most)))
    table = bool(prompt) and rng.random() < 0.5
    return _forward(None, views, prompt, table, chunk, steps, episodes)


# ------------------------------------------------------------------------------------------------ what a program keeps
@functools.lru_cache(maxsize=1)
def _checkpoint():
    return random_checkpoint(prompt_len=0, wscale=0.02, seed=0, device="cuda")


@functools.lru_cache(maxsize=1)
def _embedding_table():
    gen = torch.Generator(device="cuda").manual_seed(1)
    return (torch.randn(VOCAB_ROWS, spec.ENCODER_DIM, device="cuda", generator=gen) * 0.02).to(bf16)


def _weights(prompt):
    weights = dict(_checkpoint())
    gen = torch.Generator(device="cuda").manual_seed(2)
    weights["language_embeds"] = (torch.randn(prompt, spec.ENCODER_DIM, device="cuda", generator=gen) * 0.02).to(bf16)
    return weights


@functools.lru_cache(maxsize=2)
def _engine(views, prompt, table, chunk, steps, episodes):
    return Pi0Inference(_weights(prompt), num_views=views, chunk_size=chunk, steps=steps, episodes=episodes,
                        embedding_table=_embedding_table() if table else None)


def _randn(gen, *shape):
    return torch.randn(shape, device="cuda", generator=gen).to(bf16)


def _images(gen, *lead):
    return (torch.rand(lead + (224, 224, 3), device="cuda", generator=gen) * 2.0 - 1.0).to(bf16)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "forward":
        lead = (case["episodes"],) if case["episodes"] > 1 else ()
        s = {"engine": _engine(case["views"], case["prompt"], case["table"], case["chunk"], case["steps"], case["episodes"]),
             "images": _images(gen, *lead, case["views"]), "state": _randn(gen, *lead, spec.ACTION_DIM),
             "noise": _randn(gen, *lead, case["chunk"], spec.ACTION_DIM)}
        if case["table"]:
            s["ids"] = torch.randint(0, VOCAB_ROWS, (case["prompt"],), device="cuda", generator=gen)
        return dict(s, kind=kind)
    if kind in ("decoder_ffn", "encoder_ffn"):
        stack = kind.split("_")[0]
        dim, ffn = (spec.DECODER_DIM, spec.DECODER_FFN) if stack == "decoder" else (spec.ENCODER_DIM, spec.ENCODER_FFN)
        rows = case["tokens"]
        w = _checkpoint()
        return {"kind": kind, "ops": op_table(), "pool": ScratchPool(), "x": _randn(gen, rows, dim),
                "residual": _randn(gen, rows, dim), "hidden": torch.zeros(rows, ffn, dtype=bf16, device="cuda"),
                "out": torch.zeros(rows, dim, dtype=bf16, device="cuda"), "norm": torch.zeros(rows, dim, dtype=bf16, device="cuda"),
                "factor": torch.zeros(rows, dtype=bf16, device="cuda"),
                "w": [w[f"{stack}_ffn_{part}_w"][seed % spec.ENCODER_LAYERS] for part in ("gate", "up", "down")]}
    chunk = case.get("chunk", 50)
    buffers, S = allocate_static_buffers(case["views"], chunk, case["prompt"], "cuda")
    s = {"kind": kind, "ops": op_table(), "pool": ScratchPool(), "buffers": buffers, "S": S, "views": case["views"],
         "weights": _weights(case["prompt"])}
    if kind == "prefill":
        buffers["observation_images_normalized"].copy_(_images(gen, case["views"]))
        return s
    wrappers.register_bf16_shadow(buffers["decoder_x"], buffers["decoder_x_bf16"])
    for cache in ("encoder_K", "encoder_V"):
        buffers[cache][:, :S].copy_(_randn(gen, spec.ENCODER_LAYERS, S, spec.HEAD_DIM))
    buffers["observation_state_normalized"].copy_(_randn(gen, spec.ACTION_DIM))
    return dict(s, noise=_randn(gen, chunk, spec.ACTION_DIM), steps=case["steps"])


def run(s):
    kind = s["kind"]
    if kind == "forward":
        engine = s["engine"]
        if "ids" in s:
            engine.set_prompt(s["ids"])
        actions = engine.forward(s["images"], s["state"], s["noise"])
        return {"actions": actions, "K": [b["encoder_K"] for b in engine.episode_buffers],
                "V": [b["encoder_V"] for b in engine.episode_buffers]}
    with wrappers.use_pool(s["pool"]):
        ops = s["ops"]
        if kind == "decoder_ffn":
            s["out"].copy_(s["residual"])
            ops.decoder_norm_gated_ffn(s["x"], s["w"][0], s["w"][1], s["hidden"], s["factor"])
            ops.decoder_ffn_down_residual(s["hidden"], s["w"][2], s["out"])
            return {"hidden": s["hidden"], "out": s["out"]}
        if kind == "encoder_ffn":
            s["out"].copy_(s["residual"])
            ops.encoder_norm_gated_ffn(s["x"], s["w"][0], s["w"][1], s["hidden"], s["norm"])
            ops.encoder_ffn_down_residual(s["hidden"], s["w"][2], s["out"])
            return {"hidden": s["hidden"], "out": s["out"]}
        b = s["buffers"]
        if kind == "prefill":
            b["encoder_x"][s["views"] * spec.VISION_TOKENS:].copy_(s["weights"]["language_embeds"])
            pipeline.vision_encoder(ops, s["weights"], b, s["views"])
            pipeline.transformer_encoder(ops, s["weights"], b, s["S"])
            return {"K": b["encoder_K"], "V": b["encoder_V"]}
        b["diffusion_noise"].copy_(s["noise"])
        pipeline.transformer_decoder(ops, s["weights"], b, s["S"], steps=s["steps"])
        return {"actions": b["diffusion_noise"], "K": b["encoder_K"], "V": b["encoder_V"]}


# ------------------------------------------------------------------------------------------------ what a pass has to do
def _prefix_work(views, prompt):
    """(parameters read, flops of one episode) of SigLIP and the prefix encoder; its last layer stops after QKV."""
    T, S = views * spec.VISION_TOKENS, views * spec.VISION_TOKENS + prompt
    D, F, E, G = spec.VISION_DIM, spec.VISION_FFN, spec.ENCODER_DIM, spec.ENCODER_FFN
    patch, tower = spec.PATCH_FEATURES * D, spec.VISION_LAYERS * (4 * D * D + 2 * D * F)
    qkv, rest = spec.ENCODER_LAYERS * E * spec.QKV_DIM, (spec.ENCODER_LAYERS - 1) * (E * E + 3 * E * G)
    flops = 2.0 * T * (patch + tower + D * E) + 2.0 * S * (qkv + rest)
    flops += spec.VISION_LAYERS * 4.0 * T * spec.VISION_TOKENS * D + (spec.ENCODER_LAYERS - 1) * 4.0 * S * S * E
    return patch + tower + D * E + qkv + rest, flops


def _decoder_work(S, chunk, steps):
    """(parameters read, flops of one episode) of the action expert."""
    D, F, A = spec.DECODER_DIM, spec.DECODER_FFN, spec.DECODER_HEADS * spec.HEAD_DIM
    layer, io = D * spec.QKV_DIM + A * D + 3 * D * F, D * D + 3 * spec.ACTION_DIM * D
    rows = chunk + 1
    flops = steps * (2.0 * rows * spec.ENCODER_LAYERS * layer + 2.0 * chunk * io + spec.ENCODER_LAYERS * 4.0 * rows * (S + rows) * A)
    return spec.ENCODER_LAYERS * layer + io, flops


def work(case):
    """Every parameter and input once, every output once. (The action expert's weights, 0.6 GB, are needed again in every
    Euler step and fit no cache; here they count once all the same.)"""
    kind = case["kind"]
    if kind in ("decoder_ffn", "encoder_ffn"):
        dim, ffn = (spec.DECODER_DIM, spec.DECODER_FFN) if kind == "decoder_ffn" else (spec.ENCODER_DIM, spec.ENCODER_FFN)
        rows = case["tokens"]
        return {"bytes": 2.0 * (3 * dim * ffn + rows * (3 * dim + ffn)), "flops": 6.0 * rows * dim * ffn}
    S, chunk = case["views"] * spec.VISION_TOKENS + case["prompt"], case.get("chunk", 50)
    episodes = case.get("episodes", 1)
    params, flops, moved = 0, 0.0, 0.0
    if kind != "decode":
        params, flops = _prefix_work(case["views"], case["prompt"])
        moved += case["views"] * 224 * 224 * 3 + case["prompt"] * spec.ENCODER_DIM
    if kind != "prefill":
        p, f = _decoder_work(S, chunk, case["steps"])
        params, flops = params + p, flops + f
        moved += 2 * chunk * spec.ACTION_DIM + spec.ACTION_DIM
    moved += 2 * spec.ENCODER_LAYERS * (S + chunk + 1) * spec.HEAD_DIM          # the KV caches that come back
    return {"bytes": 2.0 * (params + episodes * moved), "flops": episodes * flops}


def tolerance(case):
    """bf16 operands and activations with fp32 accumulation: one projection is good to a few roundings; through the 27 + 18
    layers of the prefix on random weights, or a softmax over unit-variance keys, roundings grow: the two op tables of
    this package (row norms inside the GEMM against a kernel of their own) differ by 1.2e-2 in the cache rows, 1.7e-2 in
    the last layer's, with single values up to 0.1 of the rms."""
    if case["kind"] in ("decoder_ffn", "encoder_ffn"):
        return {"rel": 6e-3, "max": 4e-2}
    return {"rel": 2e-2, "max": 0.25}
