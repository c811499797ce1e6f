"""The decoder's cluster GEMM beyond 64 rows (128 token slots): the edges of its range, one sequence and several."""
from __future__ import annotations

import pytest
import torch

from conftest import assert_close
from oracle import pi0_ref as O

pytestmark = pytest.mark.gpu
bf16 = torch.bfloat16


def rnd(gen, *shape, scale=1.0):
    return (torch.randn(*shape, generator=gen) * scale).to(bf16)


# 64 | 65: the last shape of 64 slots and the first of 128; 102 = two episodes of 51; 128: every slot a row
@pytest.mark.parametrize("M,group", [(64, 0), (65, 0), (102, 51), (120, 8), (128, 64)])
def test_decoder_gemms_by_row_count(M, group):
    from flash_vla_b200 import op_table
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import _lib, wrappers
    ops, ref_ops = op_table(False), O.op_table(False)
    g = torch.Generator().manual_seed(M)
    x32 = torch.randn(M, 1024, generator=g) * 3.0
    x = x32.cuda()
    shadow = torch.zeros(M, 1024, dtype=bf16, device="cuda")
    wrappers.register_bf16_shadow(x, shadow)
    xr = x32.to(bf16).float()

    D, E, S = group or M, M // (group or M), 24
    w, rope = rnd(g, 1024, 2560, scale=0.02), O.rope_table(D, S)
    cache = torch.zeros(2, E, S + D, 256, dtype=bf16, device="cuda")
    Q, nf = torch.zeros(M * 8, 256, dtype=bf16, device="cuda"), torch.zeros(M, dtype=bf16, device="cuda")
    K, V = (c[:, S:] if group else c[0, S:] for c in cache)
    ops.decoder_norm_qkv_rope(x, w.cuda(), rope.cuda(), Q, K, V, nf)
    for e in range(E):
        refs = [torch.zeros(D * 8, 256), torch.zeros(D, 256), torch.zeros(D, 256), torch.zeros(D)]
        ref_ops.decoder_norm_qkv_rope(xr[e * D:(e + 1) * D], w.float(), rope.float(), *refs)
        got = (Q.view(E, D * 8, 256)[e], cache[0, e, S:], cache[1, e, S:], nf[e * D:(e + 1) * D])
        for a, b, what in zip(got, refs, "Q K V factor".split()):
            assert_close(a, b, what=f"decoder_norm_qkv_rope.{what}, sequence {e}")
    assert (cache[:, :, :S] == 0).all()

    wg, wu = rnd(g, 1024, 4096, scale=0.02), rnd(g, 1024, 4096, scale=0.02)
    ref, out = torch.zeros(M, 4096), torch.zeros(M, 4096, dtype=bf16, device="cuda")
    ref_ops.decoder_norm_gated_ffn(xr, wg.float(), wu.float(), ref, torch.zeros(M))
    ops.decoder_norm_gated_ffn(x, wg.cuda(), wu.cuda(), out, nf)
    assert_close(out, ref, what="decoder_norm_gated_ffn")

    for name, Kd in (("decoder_out_proj_residual", 2048), ("decoder_ffn_down_residual", 4096)):
        a, w2 = rnd(g, M, Kd), rnd(g, Kd, 1024, scale=0.02)
        ref = x.cpu().clone()
        getattr(ref_ops, name)(a.float(), w2.float(), ref)
        getattr(ops, name)(a.cuda().view(E, D, Kd) if group else a.cuda(), w2.cuda(), x.view(E, D, 1024) if group else x)
        assert_close(x, ref, what=name)
        assert torch.equal(shadow, x.to(bf16)), name
    assert _lib.load().fvla_device_status(None) == 0


# token slots: 32 up to 32 rows, 64 to 64, 96 to 96, then 128; activation tiles of 8, 16, 32, 40, 72, 80, 96 and 104 rows, seven k-blocks of the
# largest cluster in shared memory at a time, six (96 rows) and five
@pytest.mark.parametrize("M,group", [(1, 0), (11, 0), (32, 0), (33, 0), (72, 0), (73, 0), (96, 0), (96, 32), (97, 0)])
def test_decoder_gemms_by_token_slots(M, group):
    test_decoder_gemms_by_row_count(M, group)


# one key tile of 128 per CTA and two; 4 CTAs per cluster and more; a single token; two episodes that are resident together
@pytest.mark.parametrize("tokens,S,episodes", [(1, 40, 1), (11, 273, 1), (51, 816, 1), (65, 817, 1), (64, 1280, 1), (51, 768, 2), (5, 1024, 2)])
def test_decoder_attention_by_shape(tokens, S, episodes):
    from flash_vla_b200 import op_table
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import _lib
    g = torch.Generator().manual_seed(tokens * S)
    keys = S + tokens
    Q, K, V = rnd(g, episodes, tokens * 8, 256), rnd(g, episodes, keys, 256), rnd(g, episodes, keys, 256)
    q = Q.cuda().clone().view(-1, 256)
    k, v = (t.cuda() if episodes > 1 else t[0].cuda() for t in (K, V))
    op_table(True).decoder_attention(q, k, v, None, q, S)                    # out aliases Q
    for e in range(episodes):
        ref = torch.zeros(tokens * 8, 256)
        O.op_table(True).decoder_attention(Q[e].float(), K[e].float(), V[e].float(), None, ref, S)
        assert_close(q.view(episodes, -1, 256)[e], ref, what=f"decoder_attention, episode {e}")
    assert _lib.load().fvla_device_status(None) == 0


# prefix QKV with the row norm inside the GEMM by tile width: 64 columns up to 384 rows, 128 up to 896, 192 (the only width whose last
# column tile is ragged) up to 1 280, 256 up to 1 792, and past it, where the norm is a kernel of its own
@pytest.mark.parametrize("S", [257, 384, 385, 769, 896, 897, 1000, 1280, 1281, 1792, 1793])
def test_prefix_qkv_by_tile_width(S):
    from flash_vla_b200 import op_table
    g = torch.Generator().manual_seed(S)
    x, w, rope = rnd(g, S, 2048, scale=2.0), rnd(g, 2048, 2560, scale=0.02), O.rope_table(S, 0)
    outs = []
    for fused in (True, False):
        Q, K, V = (torch.zeros(n, 256, dtype=bf16, device="cuda") for n in (S * 8, S, S))
        op_table(fused).encoder_norm_qkv_rope(x.cuda(), w.cuda(), rope.cuda(), Q, K, V, torch.zeros(S, 2048, dtype=bf16, device="cuda"))
        outs.append((Q, K, V))
    refs = [torch.zeros(S * 8, 256), torch.zeros(S, 256), torch.zeros(S, 256)]
    O.op_table(False).encoder_norm_qkv_rope(x.float(), w.float(), rope.float(), *refs, torch.zeros(S, 2048))
    for got in outs:
        for a, b, what in zip(got, refs, "Q K V".split()):
            assert_close(a, b, rtol=2e-2, atol_rms=4e-2, what=f"encoder_norm_qkv_rope.{what}")


# a batch's residual projection: groups per episode in one launch or several, and regrouped into up to 128 rows
@pytest.mark.parametrize("episodes,rows,K", [(3, 51, 2048), (4, 51, 4096), (5, 51, 4096), (8, 51, 2048), (8, 51, 4096), (7, 23, 4096), (3, 127, 2048)])
def test_batched_residual_projection(episodes, rows, K):
    from flash_vla_b200 import op_table
    g = torch.Generator().manual_seed(episodes * rows)
    x, w, out = rnd(g, episodes, rows, K), rnd(g, K, 1024, scale=0.02), torch.randn(episodes, rows, 1024, generator=g)
    ref, got = out.view(-1, 1024).clone(), out.cuda()
    O.op_table(False).decoder_ffn_down_residual(x.float().view(-1, K), w.float(), ref)
    op_table(True).decoder_ffn_down_residual(x.cuda(), w.cuda(), got)
    assert_close(got.view(-1, 1024), ref, what="decoder_ffn_down_residual")


# groups of 65 rows and more, K = 4 096 in one launch: sixteen k-blocks per CTA through a ring of seven, six and five places
@pytest.mark.parametrize("episodes,rows", [(2, 72), (3, 96), (4, 97), (3, 127), (4, 128)])
def test_batched_down_projection_in_one_launch(episodes, rows):
    test_batched_residual_projection(episodes, rows, 4096)


# prefix projections beyond one round of tiles: pair tiles with K split over two rounds of items, 192-wide tiles in one and two rounds
@pytest.mark.parametrize("op,S,K", [("encoder_ffn_down_residual", 1281, 16384), ("encoder_out_proj_residual", 1281, 2048), ("encoder_out_proj_residual", 2449, 2048)])
def test_prefix_projection_by_row_count(op, S, K):
    from flash_vla_b200 import op_table
    g = torch.Generator().manual_seed(S)
    x, w, out = rnd(g, S, K), rnd(g, K, 2048, scale=0.02), rnd(g, S, 2048)
    ref, got = out.float(), out.cuda()
    getattr(O.op_table(False), op)(x.float(), w.float(), ref)
    getattr(op_table(True), op)(x.cuda(), w.cuda(), got)
    assert_close(got, ref, what=op)


# gated FFN on single SMs (one row tile, three) and on pairs (two, five), at the edges of the row tiles
@pytest.mark.parametrize("S", [65, 128, 256, 257, 384, 513, 640])
def test_prefix_gated_ffn_by_row_count(S):
    from flash_vla_b200 import op_table
    g = torch.Generator().manual_seed(S)
    x, wg, wu = rnd(g, S, 2048), rnd(g, 2048, 16384, scale=0.02), rnd(g, 2048, 16384, scale=0.02)
    ref, got, norm = torch.zeros(S, 16384), torch.zeros(S, 16384, dtype=torch.bfloat16, device="cuda"), torch.zeros(S, 2048)
    O.op_table(False).encoder_norm_gated_ffn(x.float(), wg.float(), wu.float(), ref, norm)
    op_table(True).encoder_norm_gated_ffn(x.cuda(), wg.cuda(), wu.cuda(), got, norm.bfloat16().cuda())
    assert_close(got, ref, rtol=2e-2, atol_rms=4e-2, what="encoder_norm_gated_ffn")


# a batch of episodes takes no scratch, whichever kernel serves it
@pytest.mark.parametrize("episodes", [2, 5])
def test_batched_decoder_attention_without_scratch(episodes):
    from flash_vla_b200 import op_table
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import _lib
    g, tokens, S = torch.Generator().manual_seed(episodes), 51, 768
    q, k, v = (rnd(g, episodes, n, 256).cuda() for n in (tokens * 8, S + tokens, S + tokens))
    want, got = q.view(-1, 256).clone(), torch.zeros_like(q)
    op_table(True).decoder_attention(want, k, v, None, want, S)
    _lib.call("fvla_decoder_attention", q.data_ptr(), k.data_ptr(), v.data_ptr(), got.data_ptr(), tokens * 8, S + tokens, 256, 8, S, episodes,
              tokens * 8 * 256, (S + tokens) * 256, None, 0, torch.cuda.current_stream().cuda_stream)
    assert torch.equal(got.view(-1, 256), want)


# a batch reads nothing that the kernel before it in the stream writes, the prefix rows among it, before that kernel has ended
@pytest.mark.parametrize("episodes", [2, 5])
def test_batched_decoder_attention_behind_the_kernel_that_writes_its_prefix(episodes):
    from flash_vla_b200 import op_table
    g, ops, tokens, S = torch.Generator().manual_seed(episodes), op_table(True), 51, 256
    x, w, rope = rnd(g, episodes * S, 2048).cuda(), rnd(g, 2048, 2560, scale=0.02).cuda(), O.rope_table(S, 0).to(bf16).cuda()
    q, scratch = rnd(g, episodes * tokens * 8, 256).cuda(), torch.zeros(episodes * S * 8, 256, dtype=bf16, device="cuda")
    norm, caches = torch.zeros(episodes * S, 2048, dtype=bf16, device="cuda"), [rnd(g, episodes, S + tokens, 256).cuda() for _ in range(2)]
    results = [torch.zeros_like(q), torch.zeros_like(q)]
    for wait, out in zip((True, False), results):
        for cache in caches:
            cache[:, :S] = 0
        torch.cuda.synchronize()
        ops.encoder_norm_qkv_rope(x, w, rope, scratch, caches[0][:, :S], caches[1][:, :S], norm)
        if wait:
            torch.cuda.synchronize()
        ops.decoder_attention(q, *caches, None, out, S)
    assert torch.equal(*results)


# a batch's QKV projection behind its row-norm kernel: 128-wide tiles in one round (153 and 867 rows), 256-wide ones beyond 896 rows (918, a ragged last tile)
@pytest.mark.parametrize("episodes,tokens", [(3, 51), (17, 51), (18, 51), (9, 127)])
def test_batched_qkv_projection_by_tile_width(episodes, tokens):
    from flash_vla_b200 import op_table
    M, skip = episodes * tokens, 3
    g = torch.Generator().manual_seed(M)
    # Rows rounded to bf16: 1.7e-3 of the rms in a projection's result, and under a rotation, 5.3 standard deviations of it (9e-3) in the
    # largest of two million, and half an ulp (4e-3 of the value) for the result's own rounding: inside the default bound. (A table of normal
    # variates instead of a rotation stretches rows by up to five and does not meet it.)
    x, w, rope = torch.randn(M, 1024, generator=g), rnd(g, 1024, 2560, scale=0.02), O.rope_table(tokens, 24)
    Q, K, V = (torch.zeros(*s, 256, dtype=bf16, device="cuda") for s in ((M * 8,), (episodes, skip + tokens), (episodes, skip + tokens)))
    op_table(True).decoder_norm_qkv_rope(x.cuda(), w.cuda(), rope.cuda(), Q, K[:, skip:], V[:, skip:], torch.zeros(M, dtype=bf16, device="cuda"))
    for e in (0, episodes - 1):
        r = slice(e * tokens, (e + 1) * tokens)
        ref = torch.zeros(tokens * 8, 256), torch.zeros(tokens, 256), torch.zeros(tokens, 256)
        O.op_table(False).decoder_norm_qkv_rope(x[r].clone(), w.float(), rope.float(), *ref, torch.zeros(tokens))
        for got, want, what in zip((Q[r.start * 8:r.stop * 8], K[e, skip:], V[e, skip:]), ref, "QKV"):
            assert_close(got, want, what=f"{what} of episode {e}")
    assert not K[:, :skip].any() and not V[:, :skip].any()
