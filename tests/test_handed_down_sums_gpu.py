"""Row sums handed from kernel to kernel: every partial sum against the values it stands for, and every norm that is made of them against
the oracle's, row by row, so that a few wrong rows of a ragged tile cannot hide in a whole tensor's norm.

The projections are compared on rows that stay: with the residual projections' weights at zero, x is what it was while all its sums are written
anew, and the oracle (fp32) takes the same bf16 or fp32 rows.
"""
from __future__ import annotations

import pytest
import torch

from oracle import pi0_ref as O

pytestmark = pytest.mark.gpu
bf16 = torch.bfloat16
REF = O.op_table(False)

# Rounding normal variates to bf16 is 1.66e-3 in the relative 2-norm (half an ulp is 2^-8 of a binade's lower end, uniform: 2^-8 / sqrt(3), over the
# rms of the values in a binade). Of a projection behind a norm the result is rounded, and one operand where the norm is folded into the weight (SigLIP) or the rows
# are those of the fp32 stream (a batch's decoder). In a gated result that operand counts in both factors and once more for GELU's slope. A row of 256 values
# scatters by 5.6 % (one standard deviation) about that: six of them on top. One of a row's 64 partial sums lost is 8e-3.
ONE, TWO, THREE, FOUR = (1.34 * n ** 0.5 * 1.66e-3 for n in (1, 2, 3, 4))


def rnd(gen, *shape, scale=1.0):
    return (torch.randn(*shape, device="cuda", generator=gen) * scale).to(bf16)


def assert_rows_near(got, ref, bound, what):
    got, ref = got.reshape(-1, got.shape[-1]).double(), ref.reshape(-1, ref.shape[-1]).double()
    dist = (got - ref).norm(dim=1) / ref.norm(dim=1)
    row = dist.argmax().item()
    assert dist[row] <= bound, f"{what}: row {row} of {len(dist)} is {dist[row]:.2e} off (median {dist.median():.2e}, bound {bound:.2e})"
    return dist.median().item()


def assert_squares(sums, x, what):
    """Entries [columns / 128][rows][4]: sums of squares of 32 columns each. Up to 32 squares and 31 additions in fp32, one after the other."""
    M, K = x.shape
    exact = x.double().pow(2).view(M, K // 32, 32).sum(2)
    got = sums.view(K // 128, M, 4).permute(1, 0, 2).reshape(M, K // 32).double()
    worst = ((got - exact).abs() / exact).max().item()
    assert worst <= 32 * 2 ** -24, f"{what}: {worst:.2e}"


def assert_sums(sums, x, what):
    """Entries [columns / 64][rows][2 x (sum, sum of squares)]."""
    M, K = x.shape
    parts = x.double().view(M, K // 32, 32)
    got = sums.view(K // 64, M, 2, 2).permute(1, 0, 2, 3).reshape(M, K // 32, 2).double()
    worst = ((got[..., 0] - parts.sum(2)).abs() / parts.abs().sum(2)).max().item(), ((got[..., 1] - parts.pow(2).sum(2)).abs() / parts.pow(2).sum(2)).max().item()
    assert max(worst) <= 32 * 2 ** -24, f"{what}: sums {worst[0]:.2e}, squares {worst[1]:.2e}"


# one and three row tiles of 256; several tiles per CTA in the wide projections (5 views) and in all (24)
@pytest.mark.parametrize("views", [1, 3, 4, 5, 24])
@pytest.mark.parametrize("stay", [True, False])
def test_tower(views, stay, monkeypatch):
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import stages, wrappers
    from flash_vla_b200.models.pi0.spec import weight_shapes
    from flash_vla_b200.runtime.cuda import ScratchPool
    monkeypatch.setattr(stages, "VISION_LAYERS", 1)
    gen = torch.Generator(device="cuda").manual_seed(views)
    w = {n: rnd(gen, *((1,) + tuple(s[1:]) if s[0] == 27 and len(s) in (2, 3) else s), scale=0.02) for n, s in weight_shapes(0).items() if n.startswith("vision_")}
    for n in ("pre_attn_norm_w", "pre_ffn_norm_w"):
        w["vision_" + n] += 1
    if stay:
        for n in ("attn_o_w", "attn_o_b", "ffn_down_w", "ffn_down_b"):
            w["vision_" + n].zero_()
    w["vision_position_embedding"][:9] += 2.0                # rows with a mean of several times their spread
    M = views * 256
    b = {n: torch.zeros(views, 256, width, dtype=bf16, device="cuda")
         for n, width in (("vision_x", 1152), ("vision_x_norm", 1152), ("vision_QKV", 3456), ("vision_attn", 1152), ("vision_hidden", 4304))}
    b["observation_images_normalized"] = (torch.rand(views, 224, 224, 3, device="cuda", generator=gen) * 2 - 1).to(bf16)
    pool = ScratchPool()
    with wrappers.use_pool(pool):
        assert stages.vision_tower(w, b, views)
    x = b["vision_x"].view(M, 1152)
    assert_sums(pool.get("vis_row_sums", (M * 72,), torch.float32, x.device), x, "vision_x")
    if not stay:
        return
    x32 = b["vision_x"].float()
    for op, norm, lin, out in (("vision_norm_qkv", "pre_attn_norm", "attn_qkv", "vision_QKV"), ("vision_norm_ffn_up", "pre_ffn_norm", "ffn_up", "vision_hidden")):
        ref = torch.zeros_like(b[out], dtype=torch.float32)
        getattr(REF, op)(x32, *(w[f"vision_{n}"][0].float() for n in (norm + "_w", norm + "_b", lin + "_w", lin + "_b")), ref, torch.zeros_like(x32))
        assert_rows_near(b[out], ref, THREE if op == "vision_norm_ffn_up" else TWO, out)


# ragged and whole row tiles of 128 and 256; K split in clusters, in pairs through scratch, not at all; one sequence and several
@pytest.mark.parametrize("rows,sequences", [(65, 1), (128, 1), (129, 1), (257, 1), (273, 1), (768, 1), (817, 1), (1124, 1), (273, 3), (816, 4), (768, 8)])
@pytest.mark.parametrize("stay", [True, False])
def test_encoder(rows, sequences, stay):
    from flash_vla_b200 import op_table
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import stages, wrappers
    from flash_vla_b200.hardware.nvidia.b200.pi0.buffers import rope_table
    from flash_vla_b200.runtime.cuda import ScratchPool
    gen, M, L = torch.Generator(device="cuda").manual_seed(rows + sequences), rows * sequences, 18
    w = {"encoder_" + n: torch.empty(L, *s, dtype=bf16, device="cuda") for n, s in (
        ("attn_qkv_w", (2048, 2560)), ("attn_o_w", (2048, 2048)), ("ffn_gate_w", (2048, 16384)), ("ffn_up_w", (2048, 16384)), ("ffn_down_w", (16384, 2048)))}
    for n, t in w.items():
        for l in (0, 1):
            t[l].copy_(rnd(gen, *t.shape[1:], scale=0.0 if stay and n in ("encoder_attn_o_w", "encoder_ffn_down_w") else 0.02))
    cache, rope = ((sequences,) if sequences > 1 else ()) + (L, rows + 5, 256), rope_table(rows, 0, 256, "cuda")
    x = rnd(gen, M, 2048)
    x[:7] *= 8.0
    b = {"encoder_x": x.clone(), "encoder_x_norm": torch.zeros(M, 2048, dtype=bf16, device="cuda"), "encoder_Q": rnd(gen, M * 8, 256),
         "encoder_attn": torch.zeros(M, 2048, dtype=bf16, device="cuda"), "encoder_hidden": torch.zeros(M, 16384, dtype=bf16, device="cuda"),
         "encoder_K": rnd(gen, *cache), "encoder_V": rnd(gen, *cache), "encoder_rope_weights": rope}
    pool = ScratchPool()
    with wrappers.use_pool(pool):
        stages.encoder_layers(w, b, rows, sequences)(0, 1)
    assert_squares(pool.get("enc_row_sums", (M * 64,), torch.float32, x.device), b["encoder_x"], "encoder_x")
    if not stay:
        return
    assert torch.equal(b["encoder_x"], x)
    K, V = (b[n][1, :rows] if sequences == 1 else b[n][:, 1, :rows] for n in ("encoder_K", "encoder_V"))
    got = {"hidden": b["encoder_hidden"], "Q": b["encoder_Q"].view(M, 2048), "K": K.reshape(M, 256), "V": V.reshape(M, 256)}
    ref = {n: torch.zeros(t.shape, device="cuda") for n, t in got.items()}
    norm = torch.zeros(M, 2048, device="cuda")
    REF.encoder_norm_gated_ffn(x.float(), w["encoder_ffn_gate_w"][0].float(), w["encoder_ffn_up_w"][0].float(), ref["hidden"], norm)
    for s in range(sequences):
        r = slice(s * rows, (s + 1) * rows)
        REF.encoder_norm_qkv_rope(x[r].float(), w["encoder_attn_qkv_w"][1].float(), rope.float(), ref["Q"][r].view(rows * 8, 256), ref["K"][r], ref["V"][r], norm[r])
    bounds = {"hidden": TWO, "Q": TWO, "K": TWO, "V": ONE}   # (the projection is rounded before the rotation too)
    medians = {n: assert_rows_near(got[n], ref[n], bounds[n], n) for n in got}
    # no further from the exact result than the table's ops, which round the normalised rows (and QKV too, beyond one round of tiles)
    ops, q, k, v = op_table(False), torch.zeros_like(b["encoder_Q"]), torch.zeros_like(got["K"]), torch.zeros_like(got["V"])
    hidden, xn = torch.zeros_like(b["encoder_hidden"]), torch.zeros_like(x)
    with wrappers.use_pool(ScratchPool()):
        ops.encoder_norm_gated_ffn(x, w["encoder_ffn_gate_w"][0], w["encoder_ffn_up_w"][0], hidden, xn)
        ops.encoder_norm_qkv_rope(x, w["encoder_attn_qkv_w"][1], rope.repeat(sequences, 1), q, k, v, xn)
    for n, t in (("hidden", hidden), ("Q", q.view(M, 2048)), ("K", k), ("V", v)):
        by_ops = ((t.double() - ref[n].double()).norm(dim=1) / ref[n].double().norm(dim=1)).median().item()
        assert medians[n] <= by_ops, f"{n}: {medians[n]:.3e} off, by ops {by_ops:.3e}"


# groups of 51, 65, 102, 128 and 23 rows
@pytest.mark.parametrize("episodes,tokens", [(3, 51), (2, 65), (8, 51), (4, 128), (7, 23)])
def test_decoder_batch(episodes, tokens):
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import stages, wrappers
    from flash_vla_b200.hardware.nvidia.b200.pi0.buffers import allocate_batched_decoder_buffers
    from flash_vla_b200.runtime.cuda import ScratchPool
    S, L, M = 256, 3, episodes * tokens
    gen = torch.Generator(device="cuda").manual_seed(M)
    w = {"decoder_" + n: rnd(gen, L, *s, scale=0.0 if n in ("attn_o_w", "ffn_down_w") else 0.02) for n, s in (
        ("attn_qkv_w", (1024, 2560)), ("attn_o_w", (2048, 1024)), ("ffn_gate_w", (1024, 4096)), ("ffn_up_w", (1024, 4096)), ("ffn_down_w", (4096, 1024)))}
    d = allocate_batched_decoder_buffers(tokens - 1, episodes, S, "cuda")
    x = torch.randn(M, 1024, device="cuda", generator=gen) * 3
    x[:5] *= 20
    d["decoder_x"].copy_(x)
    kv = {n: rnd(gen, episodes, L, S + tokens, 256, scale=0.5) for n in ("encoder_K", "encoder_V")}
    with wrappers.use_pool(ScratchPool()):
        run = stages.decoder_batch_layers(w, kv, d, S, episodes, L)
        run(0, 1)
        run(1, 2)                                            # a layer whose QKV projection has its norm from handed-down sums
    assert torch.equal(d["decoder_x"], x)
    hidden, rope = torch.zeros(M, 4096, device="cuda"), d["decoder_rope_weights"].float()
    REF.decoder_norm_gated_ffn(x, w["decoder_ffn_gate_w"][1].float(), w["decoder_ffn_up_w"][1].float(), hidden, torch.zeros(M, device="cuda"))
    assert_rows_near(d["decoder_hidden"], hidden, FOUR, "hidden")
    for e in range(episodes):
        q, k, v = torch.zeros(tokens * 8, 256, device="cuda"), torch.zeros(tokens, 256, device="cuda"), torch.zeros(tokens, 256, device="cuda")
        REF.decoder_norm_qkv_rope(x[e * tokens:(e + 1) * tokens].clone(), w["decoder_attn_qkv_w"][1].float(), rope, q, k, v, torch.zeros(tokens, device="cuda"))
        assert_rows_near(kv["encoder_K"][e, 1, S:], k, TWO, f"K of episode {e}")
        assert_rows_near(kv["encoder_V"][e, 1, S:], v, TWO, f"V of episode {e}")
