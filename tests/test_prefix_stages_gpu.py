"""The prefix stages that the library issues as one call (`vision_tower`, `encoder_layers`): row norms taken from sums that the
kernels before leave behind, against the oracle's ops in fp32 and against the table's own ops one by one.

Sizes: one, three and more row tiles of 128 and of 256, ragged last tiles, one tile and several per CTA, one sequence and several.
"""
from __future__ import annotations

import pytest
import torch

from conftest import assert_close
from oracle import pi0_ref as O

pytestmark = pytest.mark.gpu
bf16 = torch.bfloat16


def rnd(gen, *shape, scale=1.0):
    return (torch.randn(*shape, device="cuda", generator=gen) * scale).to(bf16)


def assert_near(got, ref, what):
    """Relative 2-norm. A result behind up to ten bf16 roundings (1.66e-3 each for normal variates, operands and stored activations) is
    5.2e-3 from the exact one, two such results are 7.4e-3 from one another; a third more is allowed."""
    got, ref = got.double(), ref.double().to(got.device)
    assert torch.isfinite(got).all(), what
    dist = ((got - ref).norm() / ref.norm()).item()
    assert dist <= 1e-2, f"{what}: relative distance {dist:.2e}"


def vision_weights(gen, layers):
    from flash_vla_b200.models.pi0.spec import weight_shapes
    w = {}
    for name, shape in weight_shapes(0).items():
        if name.startswith("vision_"):
            w[name] = rnd(gen, *((layers,) + tuple(shape[1:]) if shape[0] == 27 and len(shape) in (2, 3) else shape), scale=0.02)
    for n in ("pre_attn_norm_w", "pre_ffn_norm_w"):
        w["vision_" + n] = w["vision_" + n] + 1
    return w


@pytest.mark.parametrize("views,layers", [(1, 1), (3, 1), (24, 1), (1, 2), (3, 2), (4, 2), (12, 2), (24, 2)])
def test_vision_tower(views, layers, monkeypatch):
    """One layer takes its sums from the patch embedding, the second from the FFN. 24 views give a CTA several tiles in every
    projection. One layer: rows with a mean of many times their spread check E[x^2] - mean^2 (the rows themselves are the same on both sides)."""
    from flash_vla_b200 import op_table
    from flash_vla_b200.hardware.nvidia.b200.pi0 import pipeline
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import stages, wrappers
    from flash_vla_b200.runtime.cuda import ScratchPool
    monkeypatch.setattr(stages, "VISION_LAYERS", layers)
    monkeypatch.setattr(pipeline, "VISION_LAYERS", layers)
    gen = torch.Generator(device="cuda").manual_seed(views)
    w = vision_weights(gen, layers)
    if layers == 1:
        w["vision_position_embedding"][:32] += 4.0
    b = {n: torch.zeros(views, 256, width, dtype=bf16, device="cuda")
         for n, width in (("vision_x", 1152), ("vision_x_norm", 1152), ("vision_QKV", 3456), ("vision_attn", 1152), ("vision_hidden", 4304))}
    b["observation_images_normalized"] = (torch.rand(views, 224, 224, 3, device="cuda", generator=gen) * 2 - 1).to(bf16)
    with wrappers.use_pool(ScratchPool()):
        assert stages.vision_tower(w, b, views)
        got = {n: b[n].clone() for n in ("vision_x", "vision_QKV", "vision_hidden")}
        assert (b["vision_x_norm"] == 0).all(), "the stage must not write vision_x_norm"
        by_op = op_table(True)
        del by_op.vision_tower
        pipeline.vision_encoder(by_op, w, b, views)
    for n, t in got.items():
        if layers == 1 and n == "vision_QKV":
            assert_close(t, b[n].float().cpu(), rtol=2e-2, atol_rms=2e-2, what=n)      # either side may be an op's bound from the exact value
        assert_near(t, b[n], f"{n} against the ops")
    few = min(views, 3)                                      # the oracle: views do not depend on one another
    ref = {"vision_x": torch.zeros(few, 256, 1152), "vision_x_norm": torch.zeros(few, 256, 1152), "vision_QKV": torch.zeros(few, 256, 3456),
           "vision_attn": torch.zeros(few, 256, 1152), "vision_hidden": torch.zeros(few, 256, 4304),
           "observation_images_normalized": b["observation_images_normalized"][views - few:].float().cpu()}
    if layers == 2:
        pipeline.vision_encoder(O.op_table(True), {n: t.float().cpu() for n, t in w.items()}, ref, few)
        for n in ("vision_x", "vision_hidden"):
            assert_near(got[n][views - few:], ref[n], f"{n} against the oracle")


@pytest.mark.parametrize("rows,sequences", [(256, 1), (273, 1), (768, 1), (817, 1), (1124, 1), (256, 2), (273, 3), (768, 2), (816, 4), (768, 8)])
def test_encoder_layers(rows, sequences):
    """Layers 0 and 1 behind layer 0's QKV projection (the sums of the stage's residual projections feed layer 0's FFN, layer 1's
    projection and layer 1's FFN), then the last FFN and projection, which leave x_norm as the ops do."""
    from flash_vla_b200 import op_table
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import stages, wrappers
    from flash_vla_b200.hardware.nvidia.b200.pi0.buffers import rope_table
    from flash_vla_b200.runtime.cuda import ScratchPool
    gen, M, L = torch.Generator(device="cuda").manual_seed(rows + sequences), rows * sequences, 18
    w = {"encoder_" + n: torch.empty(L, *s, dtype=bf16, device="cuda") for n, s in (
        ("attn_qkv_w", (2048, 2560)), ("attn_o_w", (2048, 2048)), ("ffn_gate_w", (2048, 16384)), ("ffn_up_w", (2048, 16384)), ("ffn_down_w", (16384, 2048)))}
    for t in w.values():
        for l in (0, 1, 2, 16, 17):
            t[l].copy_(rnd(gen, *t.shape[1:], scale=0.02))
    cache = ((sequences,) if sequences > 1 else ()) + (L, rows + 5, 256)
    x = rnd(gen, M, 2048)
    x[:7] += 3.0

    def plan():
        return {"encoder_x": x.clone(), "encoder_x_norm": torch.zeros(M, 2048, dtype=bf16, device="cuda"),
                "encoder_Q": torch.zeros(M * 8, 256, dtype=bf16, device="cuda"), "encoder_attn": torch.zeros(M, 2048, dtype=bf16, device="cuda"),
                "encoder_hidden": torch.zeros(M, 16384, dtype=bf16, device="cuda"), "encoder_K": torch.zeros(cache, dtype=bf16, device="cuda"),
                "encoder_V": torch.zeros(cache, dtype=bf16, device="cuda"), "encoder_rope_weights": rope_table(rows, 0, 256, "cuda")}

    ops = op_table(True)

    def kv(b, layer):
        return (b["encoder_K"][layer, :rows], b["encoder_V"][layer, :rows]) if sequences == 1 else (b["encoder_K"][:, layer, :rows], b["encoder_V"][:, layer, :rows])

    def by_ops(b, first, last):
        for l in range(first, last):
            k, v = kv(b, l)
            for e in range(sequences):
                r = slice(e * rows, (e + 1) * rows)
                ops.encoder_attention(b["encoder_Q"][e * rows * 8:(e + 1) * rows * 8], k if sequences == 1 else k[e], v if sequences == 1 else v[e], 256 ** -0.5, b["encoder_attn"][r])
            ops.encoder_out_proj_residual(b["encoder_attn"], w["encoder_attn_o_w"][l], b["encoder_x"])
            ops.encoder_norm_gated_ffn(b["encoder_x"], w["encoder_ffn_gate_w"][l], w["encoder_ffn_up_w"][l], b["encoder_hidden"], b["encoder_x_norm"])
            ops.encoder_ffn_down_residual(b["encoder_hidden"], w["encoder_ffn_down_w"][l], b["encoder_x"])
            ops.encoder_norm_qkv_rope(b["encoder_x"], w["encoder_attn_qkv_w"][l + 1], b["encoder_rope_weights"], b["encoder_Q"], *kv(b, l + 1), b["encoder_x_norm"])

    with wrappers.use_pool(ScratchPool()):
        got, want = plan(), plan()
        for b, run in ((got, stages.encoder_layers(w, got, rows, sequences)), (want, lambda f, l: by_ops(want, f, l))):
            assert run is not None
            ops.encoder_norm_qkv_rope(b["encoder_x"], w["encoder_attn_qkv_w"][0], b["encoder_rope_weights"], b["encoder_Q"], *kv(b, 0), b["encoder_x_norm"])
            run(0, 1)
            b["one"] = b["encoder_hidden"].clone()
            run(1, 2)
            b["two"] = b["encoder_hidden"].clone()
        for n in ("one", "two", "encoder_x", "encoder_Q", "encoder_K", "encoder_V"):
            assert_near(got[n], want[n], n)
        # the last FFN and projection, which leave x_norm
        run = stages.encoder_layers(w, got, rows, sequences)
        for b in (got, want):
            b["encoder_x"].copy_(x)
            ops.encoder_norm_qkv_rope(b["encoder_x"], w["encoder_attn_qkv_w"][16], b["encoder_rope_weights"], b["encoder_Q"], *kv(b, 16), b["encoder_x_norm"])
        run(16, 17)
        by_ops(want, 16, 17)
        for n in ("encoder_x", "encoder_x_norm", "encoder_hidden", "encoder_Q"):
            assert_near(got[n], want[n], n + " of the last layer")


def test_frozen_pool_and_pinned_plans_go_op_by_op():
    """A pool frozen before the stage ever ran, and a pinned launch plan, are served by the ops as before."""
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import _lib, stages, wrappers
    from flash_vla_b200.runtime.cuda import ScratchPool
    gen = torch.Generator(device="cuda").manual_seed(0)
    w = vision_weights(gen, 27)
    b = {n: torch.zeros(1, 256, width, dtype=bf16, device="cuda")
         for n, width in (("vision_x", 1152), ("vision_x_norm", 1152), ("vision_QKV", 3456), ("vision_attn", 1152), ("vision_hidden", 4304))}
    b["observation_images_normalized"] = torch.zeros(1, 224, 224, 3, dtype=bf16, device="cuda")
    pool = ScratchPool()
    pool.freeze()
    with wrappers.use_pool(pool):
        assert not stages.vision_tower(w, b, 1)
    with wrappers.use_pool(ScratchPool()):
        assert stages.vision_tower(w, b, 1)
        _lib.call("fvla_gemm_plan_set", 256, 1152, 1152, 0, 1, 64, 1)
        try:
            assert not stages.vision_tower(w, b, 1)
        finally:
            _lib.call("fvla_gemm_plan_clear")


@pytest.mark.parametrize("views", [4, 5, 9, 12, 24])
def test_vision_attention_by_views(views):
    """One query half per CTA (4 and 12 views) and both: a view's result does not depend on its neighbours or on the form."""
    from flash_vla_b200 import op_table
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import _lib
    gen = torch.Generator(device="cuda").manual_seed(views)
    qkv = rnd(gen, views, 256, 3456)
    qkv[:, :9] *= 25.0                                       # some rows whose softmax is all but one-hot
    ops, out = op_table(True), torch.zeros(views, 256, 1152, dtype=bf16, device="cuda")
    ops.vision_attention(qkv, out)
    for v in (0, views // 2, views - 1):
        alone = torch.zeros(1, 256, 1152, dtype=bf16, device="cuda")
        ops.vision_attention(qkv[v:v + 1].contiguous(), alone)
        assert torch.equal(out[v], alone[0]), f"view {v}"
    ref = torch.zeros(2, 256, 1152)
    O.op_table(False).vision_attention(qkv[-2:].float().cpu(), ref)
    assert_close(out[-2:], ref, what="vision_attention")
    assert _lib.load().fvla_device_status(None) == 0


def test_folded_layers_follow_the_weights():
    """The tower finds each layer's folded weights where the op keeps them, and folds again after an in-place update of any of the four stacks."""
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import wrappers
    gen = torch.Generator(device="cuda").manual_seed(0)
    w, nw, nb, b = rnd(gen, 3, 1152, 64, scale=0.02), rnd(gen, 3, 1152) + 1, rnd(gen, 3, 1152), rnd(gen, 3, 64)
    first = wrappers._folded_layers(w, nw, nb, b)
    assert all(f is g for f, g in zip(first, wrappers._folded_layers(w, nw, nb, b)))
    assert all(wrappers._folded_layernorm(w[l], nw[l], nb[l], b[l]) is first[l] for l in range(3))
    for t in (w, nw, nb, b):
        t[1].mul_(2.0)
        again = wrappers._folded_layers(w, nw, nb, b)
        for l in range(3):
            folded = (nw[l].float()[:, None] * w[l].float()).to(bf16)
            assert torch.equal(again[l][0], folded), "weight_folded"
            torch.testing.assert_close(again[l][2], nb[l].float() @ w[l].float() + b[l].float(), rtol=1e-4, atol=1e-4)      # fp32 sums of 1 152 products
