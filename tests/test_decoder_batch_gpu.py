"""A batch's decoder layers as one call of the library (`decoder_batch_layers`): RMS norms from the sums of squares that the residual
projections leave behind, against the table's own ops and against the oracle's."""
from __future__ import annotations

import pytest
import torch

from oracle import pi0_ref as O

pytestmark = pytest.mark.gpu
bf16 = torch.bfloat16


def assert_near(got, ref, what, bound):
    got, ref = got.double(), ref.double().to(got.device)
    assert torch.isfinite(got).all(), what
    dist = ((got - ref).norm() / ref.norm()).item()
    assert dist <= bound, f"{what}: relative distance {dist:.2e}"


# 153 rows: the first shape beyond two episodes of 51; 130 and 512: fewest and most rows of a group size; 408: four groups of 102; 161: groups of 23
@pytest.mark.parametrize("episodes,tokens", [(2, 65), (3, 51), (5, 51), (8, 51), (7, 23), (8, 64)])
def test_decoder_batch_layers(episodes, tokens):
    from flash_vla_b200 import op_table
    from flash_vla_b200.hardware.nvidia.b200.pi0 import pipeline
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import _lib, stages, wrappers
    from flash_vla_b200.hardware.nvidia.b200.pi0.buffers import allocate_batched_decoder_buffers
    from flash_vla_b200.runtime.cuda import ScratchPool
    S, L, M = 273, 3, episodes * tokens
    gen = torch.Generator(device="cuda").manual_seed(M)

    def rnd(*shape, scale=1.0):
        return (torch.randn(*shape, device="cuda", generator=gen) * scale).to(bf16)

    w = {"decoder_" + n: rnd(L, *s, scale=0.02) for n, s in (("attn_qkv_w", (1024, 2560)), ("attn_o_w", (2048, 1024)), ("ffn_gate_w", (1024, 4096)),
                                                             ("ffn_up_w", (1024, 4096)), ("ffn_down_w", (4096, 1024)))}
    x0 = torch.randn(M, 1024, device="cuda", generator=gen) * 3
    x0[:5] *= 20                                             # rows of very different size: the factor is per row
    kv = [rnd(episodes, L, S + tokens, 256, scale=0.5) for _ in range(2)]
    results = []
    for by_op in (False, True):
        d = allocate_batched_decoder_buffers(tokens - 1, episodes, S, "cuda")
        d["decoder_x"].copy_(x0)
        caches = {"encoder_K": kv[0].clone(), "encoder_V": kv[1].clone()}
        with wrappers.use_pool(ScratchPool()):
            ops = op_table(True)
            run = stages.decoder_batch_layers(w, caches, d, S, episodes, L)
            assert run is not None
            if by_op:
                def run(first, last):
                    x, q, nf, x3 = d["decoder_x"], d["decoder_q_buf"], d["decoder_norm_factor_buf"], d["decoder_x"].view(episodes, tokens, 1024)
                    for l in range(first, last):
                        k, v = caches["encoder_K"][:, l], caches["encoder_V"][:, l]
                        ops.decoder_norm_qkv_rope(x, w["decoder_attn_qkv_w"][l], d["decoder_rope_weights"], q, k[:, S:], v[:, S:], nf)
                        ops.decoder_attention(q, k, v, None, q, S)
                        ops.decoder_out_proj_residual(q.view(episodes, tokens, 2048), w["decoder_attn_o_w"][l], x3)
                        ops.decoder_norm_gated_ffn(x, w["decoder_ffn_gate_w"][l], w["decoder_ffn_up_w"][l], d["decoder_hidden"], nf)
                        ops.decoder_ffn_down_residual(d["decoder_hidden"].view(episodes, tokens, -1), w["decoder_ffn_down_w"][l], x3)
            seen = {}
            for l in range(L):
                run(l, l + 1)
                seen.update({f"x{l}": d["decoder_x"].clone(), f"hidden{l}": d["decoder_hidden"].clone(), f"K{l}": caches["encoder_K"][:, l, S:].clone(),
                             f"V{l}": caches["encoder_V"][:, l, S:].clone()})
            seen["factor"] = d["decoder_norm_factor_buf"].clone()
            if not by_op:
                assert torch.equal(d["decoder_x_bf16"], d["decoder_x"].to(bf16)), "shadow"
        for c, before in zip((caches["encoder_K"], caches["encoder_V"]), kv):
            assert torch.equal(c[:, :, :S], before[:, :, :S]), "prefix rows are not written"
        results.append(seen)
    # Operands rounded to bf16 on both sides (1.66e-3 each for normal variates, different values): up to twelve such roundings through
    # three layers are 5.8e-3 per side, 8.1e-3 between them; a third more
    for n, got in results[0].items():
        assert_near(got, results[1][n], n, 1.1e-2)

    # layer 0 against the oracle in fp32, an episode of its own
    ops32, e = O.op_table(False), episodes - 1
    r = slice(e * tokens, (e + 1) * tokens)
    x, q, nf = x0[r].cpu().clone(), torch.zeros(tokens * 8, 256), torch.zeros(tokens)
    k, v = kv[0][e, 0].float().cpu(), kv[1][e, 0].float().cpu()
    rope = allocate_batched_decoder_buffers(tokens - 1, episodes, S, "cuda")["decoder_rope_weights"].float().cpu()
    f = {n: t[0].float().cpu() for n, t in w.items()}
    ops32.decoder_norm_qkv_rope(x, f["decoder_attn_qkv_w"], rope, q, k[S:], v[S:], nf)
    O.op_table(True).decoder_attention(q.clone(), k, v, None, q, S)
    ops32.decoder_out_proj_residual(q.view(tokens, 2048), f["decoder_attn_o_w"], x)
    hidden = torch.zeros(tokens, 4096)
    ops32.decoder_norm_gated_ffn(x, f["decoder_ffn_gate_w"], f["decoder_ffn_up_w"], hidden, nf)
    ops32.decoder_ffn_down_residual(hidden, f["decoder_ffn_down_w"], x)
    assert_near(results[0]["hidden0"][r], hidden, "hidden against the oracle", 1e-2)
    assert_near(results[0]["x0"][r], x, "x against the oracle", 1e-2)
    assert _lib.load().fvla_device_status(None) == 0
    assert pipeline._stage(op_table(True), "decoder_batch_layers") is not None


def test_up_to_128_rows_and_wide_episodes_go_op_by_op():
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import _lib
    lib = _lib.load()
    assert [lib.fvla_decoder_batch_supported(e, t) for e, t in ((1, 200), (2, 64), (2, 129), (0, 51), (3, 0), (3, 51))] == [0, 0, 0, 0, 0, 1]


# row groups of 65, 51, 102, 128 and 23 rows; both projections, through the ring and without
@pytest.mark.parametrize("episodes,tokens", [(2, 65), (3, 51), (8, 51), (4, 128), (7, 23)])
@pytest.mark.parametrize("last", ["o", "down"])
def test_handed_down_squares_are_those_of_the_fp32_rows(episodes, tokens, last):
    """The residual stream is fp32, and so are the squares that the norms are made of: each partial sum against the 32 values it stands for."""
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import stages, wrappers
    from flash_vla_b200.hardware.nvidia.b200.pi0.buffers import allocate_batched_decoder_buffers
    from flash_vla_b200.runtime.cuda import ScratchPool
    S, L, M = 256, 1, episodes * tokens
    gen = torch.Generator(device="cuda").manual_seed(M)
    w = {"decoder_" + n: (torch.randn(L, *s, device="cuda", generator=gen) * 0.02).to(bf16) for n, s in (
        ("attn_qkv_w", (1024, 2560)), ("attn_o_w", (2048, 1024)), ("ffn_gate_w", (1024, 4096)), ("ffn_up_w", (1024, 4096)), ("ffn_down_w", (4096, 1024)))}
    if last == "o":
        w["decoder_ffn_down_w"].zero_()                      # the rows stay those of the output projection, their squares are written again
    d = allocate_batched_decoder_buffers(tokens - 1, episodes, S, "cuda")
    d["decoder_x"].copy_(torch.randn(M, 1024, device="cuda", generator=gen) * 3)
    d["decoder_x"][:5] *= 20
    kv = {n: (torch.randn(episodes, L, S + tokens, 256, device="cuda", generator=gen) * 0.5).to(bf16) for n in ("encoder_K", "encoder_V")}
    pool = ScratchPool()
    with wrappers.use_pool(pool):
        stages.decoder_batch_layers(w, kv, d, S, episodes, L)(0, L)
    sums = pool.get("dec_row_sums", (M * 32,), torch.float32, d["decoder_x"].device).view(8, M, 4).permute(1, 0, 2).reshape(M, 32)
    exact = d["decoder_x"].double().pow(2).view(M, 32, 32).sum(2)
    # 32 squares and 31 additions in fp32, half an ulp each, pairwise: 7 roundings of 2^-24. (Squares of bf16 values: up to 2^-8.)
    worst = ((sums.double() - exact).abs() / exact).max().item()
    assert worst <= 7 * 2 ** -24, worst
