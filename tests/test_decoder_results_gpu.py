"""The decoder's results up to 64 rows, bit for bit, against digests recorded on a B200 (`golden/decoder_results.json`).

Ten Euler steps on unit-variance keys multiply any difference by about 1.45 each, so a changed order of summation or a P rounded
against another maximum puts a decode further from its earlier result (0.3 in the relative 2-norm) than any tolerance allows.
Inputs are drawn on the CPU. `python tests/test_decoder_results_gpu.py` prints the digests of the library that is there."""
from __future__ import annotations

import hashlib
import json
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu
bf16 = torch.bfloat16
GOLDEN = Path(__file__).parent / "golden" / "decoder_results.json"


def rnd(gen, *shape, scale=1.0):
    return (torch.randn(*shape, generator=gen) * scale).to(bf16).cuda()


def digest(*tensors):
    h = hashlib.sha256()
    for t in tensors:
        h.update(t.detach().contiguous().cpu().view(torch.uint8).numpy().tobytes())
    return h.hexdigest()[:32]


# one row, half of the slots, an owner's slice that is not full, all 64
@pytest.fixture(params=[1, 33, 51, 64])
def rows(request):
    return request.param


def projections(M):
    from flash_vla_b200 import op_table
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import wrappers
    ops, g = op_table(True), torch.Generator().manual_seed(M)
    x, shadow = (torch.randn(M, 1024, generator=g) * 3.0).cuda(), torch.zeros(M, 1024, dtype=bf16, device="cuda")
    wrappers.register_bf16_shadow(x, shadow)
    Q, K, V = (torch.zeros(n, 256, dtype=bf16, device="cuda") for n in (M * 8, M, M))
    nf, hidden = torch.zeros(M, dtype=bf16, device="cuda"), torch.zeros(M, 4096, dtype=bf16, device="cuda")
    got = {}
    ops.decoder_norm_qkv_rope(x, rnd(g, 1024, 2560, scale=0.02), rnd(g, M, 256), Q, K, V, nf)
    got["norm_qkv_rope"] = digest(Q, K, V, nf)
    wg, wu = rnd(g, 1024, 4096, scale=0.02), rnd(g, 1024, 4096, scale=0.02)
    ops.decoder_norm_gated_ffn(x, wg, wu, hidden, nf)
    got["norm_gated_ffn"] = digest(hidden, nf)
    ops.decoder_norm_gated_ffn(torch.randn(M, 1024, generator=g).cuda(), wg, wu, hidden, nf)         # fp32 rows without a shadow
    got["norm_gated_ffn_fp32"] = digest(hidden, nf)
    ops.decoder_out_proj_residual(rnd(g, M, 2048), rnd(g, 2048, 1024, scale=0.02), x)
    got["out_proj_residual"] = digest(x, shadow)
    ops.decoder_ffn_down_residual(rnd(g, M, 4096), rnd(g, 4096, 1024, scale=0.02), x)
    got["ffn_down_residual"] = digest(x, shadow)
    ops.decoder_action_mlp(rnd(g, M, 1024), rnd(g, 1024, 1024, scale=0.02), rnd(g, 1024), x)
    got["action_mlp"] = digest(x, shadow)
    return got


def test_projections_keep_their_bits(rows):
    assert projections(rows) == json.loads(GOLDEN.read_text())[f"projections {rows}"]


# one group of 64 keys per CTA and two; ranks without keys; 8 ranges of keys and 11; the last rows of a cluster missing
ATTENTION = [(1, 40), (11, 273), (51, 768), (33, 1000), (64, 1280), (20, 1357)]


def attention(tokens, S):
    from flash_vla_b200 import op_table
    g = torch.Generator().manual_seed(tokens * S)
    q, k, v = rnd(g, tokens * 8, 256), rnd(g, S + tokens, 256), rnd(g, S + tokens, 256)
    op_table(True).decoder_attention(q, k, v, None, q, S)
    return digest(q)


@pytest.mark.parametrize("tokens,S", ATTENTION)
def test_attention_keeps_its_bits(tokens, S):
    assert attention(tokens, S) == json.loads(GOLDEN.read_text())[f"attention {tokens} {S}"]


def decoder_state(chunk, views=3, prompt=0, layers=3):
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import wrappers
    from flash_vla_b200.hardware.nvidia.b200.pi0.buffers import allocate_static_buffers
    from flash_vla_b200.models.pi0.spec import weight_shapes
    g = torch.Generator().manual_seed(chunk)
    w = {n: rnd(g, *((layers, *s[1:]) if s[0] == 18 else s), scale=0.02) for n, s in weight_shapes(0).items() if n.startswith("decoder_")}
    b, S = allocate_static_buffers(views, chunk, prompt, "cuda")
    wrappers.register_bf16_shadow(b["decoder_x"], b["decoder_x_bf16"])
    for cache in ("encoder_K", "encoder_V"):
        b[cache][:layers, :S].copy_(rnd(g, layers, S, 256))
    b["observation_state_normalized"].copy_(rnd(g, 32))
    b["diffusion_noise"].copy_(rnd(g, chunk, 32))
    return w, b, S


def decode(chunk, views, prompt, steps=10, layers=3):
    from flash_vla_b200 import op_table
    from flash_vla_b200.hardware.nvidia.b200.pi0 import pipeline
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import wrappers
    from flash_vla_b200.runtime.cuda import ScratchPool
    w, b, S = decoder_state(chunk, views, prompt, layers)
    with wrappers.use_pool(ScratchPool()):
        pipeline.transformer_decoder(op_table(True), w, b, S, steps=steps, layers=layers)
    return digest(b["diffusion_noise"], b["diffusion_noise_f32"], b["encoder_K"], b["encoder_V"])


DECODES = [(50, 3, 0), (10, 1, 17), (63, 3, 48)]


@pytest.mark.parametrize("chunk,views,prompt", DECODES)
def test_ten_euler_steps_keep_their_bits(chunk, views, prompt):
    assert decode(chunk, views, prompt) == json.loads(GOLDEN.read_text())[f"decode {chunk} {views} {prompt}"]


# the loop in native code, the ops one by one, the same with an op replaced, and buffers that the native loop does not take
@pytest.mark.parametrize("first_step", [0, 1])
@pytest.mark.parametrize("chunk", [50, 64])
def test_the_native_loop_gives_the_bits_of_its_ops(chunk, first_step):
    from flash_vla_b200 import op_table
    from flash_vla_b200.hardware.nvidia.b200.pi0 import pipeline
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import wrappers
    from flash_vla_b200.runtime.cuda import ScratchPool
    native, by_op, replaced, calls = op_table(True), op_table(True), op_table(True), []
    del by_op.decoder_steps
    replaced.decoder_attention = lambda *args: (calls.append(1), by_op.decoder_attention(*args))
    results = []
    for table, longer_rope in ((native, False), (by_op, False), (replaced, False), (native, True)):
        w, b, S = decoder_state(chunk)
        if longer_rope:
            b["decoder_rope_weights"] = torch.cat([b["decoder_rope_weights"]] * 2)
        with wrappers.use_pool(ScratchPool()):
            if first_step:
                pipeline.decoder_prologue(table, w, b)
                pipeline.decoder_step(table, w, b, S, 0, 3, noise=b["diffusion_noise_f32"])
            pipeline.transformer_decoder(table, w, b, S, steps=4, layers=3, first_step=first_step)
        results.append({n: b[n].clone() for n in ("diffusion_noise", "diffusion_noise_f32", "encoder_K", "encoder_V", "decoder_x",
                                                  "decoder_x_bf16", "decoder_norm_factor_buf")})
    assert len(calls) == 4 * 3
    for other in results[1:]:
        for name, t in results[0].items():
            assert torch.equal(t, other[name]), name


if __name__ == "__main__":
    got = {f"projections {M}": projections(M) for M in (1, 33, 51, 64)}
    got.update({f"attention {t} {S}": attention(t, S) for t, S in ATTENTION})
    got.update({f"decode {c} {v} {p}": decode(c, v, p) for c, v, p in DECODES})
    print(json.dumps(got, indent=1))
