"""Whole stages of the pipeline as one call into the library.

Not call sites of the reference's op table: `op_table(fused=True)` carries them beside the ops. A stage names the ops it
stands for (`stands_for`); `pipeline` takes it while the table still has exactly those, else it issues the table's own ops one by one.
"""
from __future__ import annotations

import ctypes

import torch

from flash_vla_b200.models.pi0.spec import ENCODER_LAYERS, VISION_LAYERS

from . import _lib, fused_wrappers
from . import wrappers as _w

_WIDTH, _QKV, _Q, _FFN, _ACT = 1024, 2560, 2048, 4096, 32


def _fits(t, shape, dtype=torch.bfloat16) -> bool:
    return isinstance(t, torch.Tensor) and t.is_cuda and t.dtype == dtype and t.shape == shape and t.is_contiguous()


def decoder_steps(weights, buffers, encoder_seq_len, steps, layers, first_step=0) -> bool:
    """Euler steps [first_step, steps) of the action expert: `pipeline.transformer_decoder` without the state projection,
    the launches of its ops issued from native code. Outside a CUDA graph a step is bound by its 93 calls otherwise:
    18 us each through the op wrappers, on the 51-row call sites that run 5 - 8 us. Returns False, having done nothing,
    for whatever is not the fp32 residual-stream plan with stacked contiguous weights and a cache of prefix + chunk + 1 rows."""
    b, w = buffers, weights
    noise, master, x, K, V = b["diffusion_noise"], b.get("diffusion_noise_f32"), b["decoder_x"], b["encoder_K"], b["encoder_V"]
    stacks = [w[f"decoder_{n}_w"] for n in ("attn_qkv", "attn_o", "ffn_gate", "ffn_up", "ffn_down")]
    if not all(isinstance(t, torch.Tensor) for t in (noise, master, x, K, V, *stacks)) or x.ndim != 2 or K.ndim != 3:
        return False
    D, total, S = x.shape[0], stacks[0].shape[0], encoder_seq_len
    chunk, rows, f32 = D - 1, K.shape[1], torch.float32
    if layers < 1 or layers > total or K.shape[0] < layers or chunk < 1 or S < 1 or first_step < 0 or steps < first_step:
        return False
    shapes = ((_WIDTH, _QKV), (_Q, _WIDTH), (_WIDTH, _FFN), (_WIDTH, _FFN), (_FFN, _WIDTH))
    small = {"in_w": (w["decoder_action_fused_in_proj_w"], (_ACT, _WIDTH)), "time_bias": (w["decoder_action_fused_time_biases"], (10, _WIDTH)),
             "mlp_w": (w["decoder_action_mlp_w"], (_WIDTH, _WIDTH)), "mlp_b": (w["decoder_action_mlp_b"], (_WIDTH,)),
             "out_w": (w["decoder_action_fused_out_proj_w"], (_WIDTH, _ACT)), "out_b": (w["decoder_action_fused_out_proj_b"], (_ACT,)),
             "rope": (b["decoder_rope_weights"], (D, 256)), "state": (b["decoder_state_buf"], (1, _WIDTH)), "noise": (noise, (chunk, _ACT)),
             "in_buf": (b["decoder_x_buf"], (chunk, _WIDTH)), "q": (b["decoder_q_buf"], (D * _w.DECODER_HEADS, 256)),
             "hidden": (b["decoder_hidden"], (D, _FFN)), "norm_factor": (b["decoder_norm_factor_buf"], (D,)),
             "k_cache": (K, (K.shape[0], S + D, 256)), "v_cache": (V, (K.shape[0], S + D, 256))}
    small.update({n: (t, (total, *s)) for n, t, s in zip(("qkv_w", "attn_o_w", "gate_w", "up_w", "down_w"), stacks, shapes)})
    if not (all(_fits(t, shape) for t, shape in small.values()) and _fits(x, (D, _WIDTH), f32) and _fits(master, (chunk, _ACT), f32)):
        return False

    def scratch(role, M, N, Kd, dual=0):
        return _w._ws(role, _lib.gemm_workspace_bytes(M, N, Kd, dual), x.device)

    ws = {"mlp": scratch("dec_mlp_ws", chunk, _WIDTH, _WIDTH), "qkv": scratch("dec_qkv_ws", D, _QKV, _WIDTH),
          "attn": _w._ws("dec_attn_ws", _lib.load().fvla_decoder_attention_workspace_bytes(D * _w.DECODER_HEADS, rows), x.device),
          "o": scratch("dec_o_ws", D, _WIDTH, _Q), "gate": scratch("dec_gate_ws", D, _FFN, _WIDTH, 1),
          "down": scratch("dec_down_ws", D, _WIDTH, _FFN)}
    args = _lib.DecoderSteps(
        noise_f32=master.data_ptr(), x=x.data_ptr(), x_shadow=_w._shadow_of(x), chunk=chunk, prefix=S, cache_rows=rows,
        first_step=first_step, steps=steps, layers=layers, **{n: t.data_ptr() for n, (t, _) in small.items()},
        **{f"ws_{k}": v[0] for k, v in ws.items()}, **{f"ws_{k}_bytes": v[1] for k, v in ws.items()})
    _lib.call("fvla_decoder_steps_run", ctypes.byref(args), _w._stream())
    return True


_VIS, _VIS_FFN, _ENC, _ENC_FFN = _w.VISION_DIM, 4304, 2048, 16384


def vision_tower(weights, buffers, num_views) -> bool:
    """`pipeline.vision_encoder` as one call: the kernels that write the residual stream leave their rows' sums behind and the
    projections take the LayerNorm from those, so that no launch reads the stream for its statistics alone. Returns False,
    having done nothing, for whatever is not the plan's contiguous buffers and stacked weights, for launch plans
    pinned by a program, and where folding a weight or a new scratch buffer would allocate while a graph is captured."""
    b, w = buffers, weights
    images, x = b["observation_images_normalized"], b["vision_x"]
    stacks = {n: w[f"vision_{n}"] for n in ("attn_qkv_w", "attn_qkv_b", "attn_o_w", "attn_o_b", "ffn_up_w", "ffn_up_b", "ffn_down_w", "ffn_down_b",
                                            "pre_attn_norm_w", "pre_attn_norm_b", "pre_ffn_norm_w", "pre_ffn_norm_b")}
    if not all(isinstance(t, torch.Tensor) for t in (images, x, *stacks.values())) or x.ndim != 3 or stacks["attn_o_w"].ndim != 3:
        return False
    V, L, D, F = x.shape[0], stacks["attn_o_w"].shape[0], _VIS, _VIS_FFN
    shapes = {"attn_qkv_w": (L, D, 3 * D), "attn_qkv_b": (L, 3 * D), "attn_o_w": (L, D, D), "attn_o_b": (L, D), "ffn_up_w": (L, D, F),
              "ffn_up_b": (L, F), "ffn_down_w": (L, F, D), "ffn_down_b": (L, D)}
    plain = {"images": (images, (V, 224, 224, 3)), "patch_w": (w["vision_patch_embedding_w"], (14, 14, 3, D)),
             "patch_b": (w["vision_patch_embedding_b"], (D,)), "pos_emb": (w["vision_position_embedding"], (_w.VISION_TOKENS, D)),
             "x": (x, (V, _w.VISION_TOKENS, D)), "qkv": (b["vision_QKV"], (V, _w.VISION_TOKENS, 3 * D)),
             "attn": (b["vision_attn"], (V, _w.VISION_TOKENS, D)), "hidden": (b["vision_hidden"], (V, _w.VISION_TOKENS, F))}
    M, dev, lib = V * _w.VISION_TOKENS, x.device, _lib.load()
    if L != VISION_LAYERS or not all(_fits(t, s) for t, s in plain.values()) or not all(_fits(t, shapes.get(n, (L, D))) for n, t in stacks.items()):
        return False
    if not lib.fvla_row_sums_supported(M):
        return False
    roles = {"sums": ("vis_row_sums", (M * (D // 32) * 2,), torch.float32), "patch": ("patches", (lib.fvla_patch_embed_workspace_bytes(V),), torch.uint8),
             "o": ("vis_o_ws", (_lib.gemm_workspace_bytes(M, D, D, 0),), torch.uint8), "down": ("vis_down_ws", (_lib.gemm_workspace_bytes(M, D, F, 0),), torch.uint8)}
    if not all(_w.scratch_covers(role, shape, dtype, dev) for role, shape, dtype in roles.values()):
        return False
    folded = [_w._folded_layers(stacks[f"{lin}_w"], stacks[f"{norm}_w"], stacks[f"{norm}_b"], stacks[f"{lin}_b"])
              for lin, norm in (("attn_qkv", "pre_attn_norm"), ("ffn_up", "pre_ffn_norm"))]
    if None in folded:
        return False
    bufs = {n: _w.scratch(role, shape, dtype, dev) for n, (role, shape, dtype) in roles.items()}
    arrays = [(ctypes.c_void_p * L)(*(f[i].data_ptr() for f in side)) for side in folded for i in range(3)]
    names = ("qkv_folded", "qkv_colsum", "qkv_bias", "up_folded", "up_colsum", "up_bias")
    args = _lib.VisionTower(
        views=V, layers=L, o_w=stacks["attn_o_w"].data_ptr(), o_b=stacks["attn_o_b"].data_ptr(), down_w=stacks["ffn_down_w"].data_ptr(),
        down_b=stacks["ffn_down_b"].data_ptr(), row_sums=bufs["sums"].data_ptr(), **{n: t.data_ptr() for n, (t, _) in plain.items()},
        **{n: ctypes.addressof(a) for n, a in zip(names, arrays)},
        **{f"ws_{n}": bufs[n].data_ptr() for n in ("patch", "o", "down")}, **{f"ws_{n}_bytes": bufs[n].numel() for n in ("patch", "o", "down")})
    return _lib.offered("fvla_vision_tower_run", ctypes.byref(args), _w._stream())


def vision_tower_as_by_op(weights, buffers, num_views) -> bool:
    """`vision_tower` for as many views as the table's own ops read folded weights for (one to four). With more they read the weights
    themselves, and a graph captured from them follows an in-place update, which one with folded copies cannot: those go op by op. (What that costs a
    forward of ten steps: two episodes of three views 13.1 -> 13.3 ms, four 23.5 -> 23.65, eight nothing beyond noise.)"""
    x = buffers["vision_x"]
    if not isinstance(x, torch.Tensor) or x.ndim != 3:
        return False
    M = x.shape[0] * _w.VISION_TOKENS
    return all(_lib.load().fvla_fused_norm_supported(M, N, _VIS, 0) for N in (3 * _VIS, _VIS_FFN)) and vision_tower(weights, buffers, num_views)


def encoder_layers(weights, buffers, rows, sequences=1):
    """The prefix encoder behind its first QKV projection: a function that enqueues layers [first, last) up to layer `last`'s QKV
    projection, or None where the ops have to be called one by one (see `vision_tower`). Row norms come from sums that the
    residual projections leave behind; a batch's attention is one launch over its sequences."""
    b, w = buffers, weights
    x, K, V = b["encoder_x"], b["encoder_K"], b["encoder_V"]
    stacks = {n: w[f"encoder_{n}"] for n in ("attn_qkv_w", "attn_o_w", "ffn_gate_w", "ffn_up_w", "ffn_down_w")}
    L, M, D, F, hd = ENCODER_LAYERS, rows * sequences, _ENC, _ENC_FFN, 256
    if not all(isinstance(t, torch.Tensor) for t in (x, K, V, *stacks.values())) or x.ndim != 2 or K.ndim != (3 if sequences == 1 else 4):
        return None
    shapes = {"attn_qkv_w": (L, D, _QKV), "attn_o_w": (L, D, D), "ffn_gate_w": (L, D, F), "ffn_up_w": (L, D, F), "ffn_down_w": (L, F, D)}
    cache = (L, K.shape[-2], hd) if sequences == 1 else (sequences, L, K.shape[-2], hd)
    plain = {"x": (x, (M, D)), "x_norm": (b["encoder_x_norm"], (M, D)), "q": (b["encoder_Q"], (M * _w.DECODER_HEADS, hd)),
             "attn": (b["encoder_attn"], (M, D)), "hidden": (b["encoder_hidden"], (M, F)), "rope": (b["encoder_rope_weights"], (rows, hd))}
    if K.shape[-2] < rows or not all(_fits(t, s) for t, s in plain.values()) or not all(_fits(stacks[n], s) for n, s in shapes.items()):
        return None
    if not _fits(K, cache) or not _fits(V, cache) or not _lib.load().fvla_row_sums_supported(M):
        return None
    u8, dev = torch.uint8, x.device
    roles = {"sums": ("enc_row_sums", (M * (D // 32),), torch.float32),
             "attn": ("enc_attn_ws", (_lib.load().fvla_encoder_attention_workspace_bytes(rows * _w.DECODER_HEADS, rows),), u8),
             "o": ("enc_o_ws", (_lib.gemm_workspace_bytes(M, D, D, 0),), u8), "down": ("enc_down_ws", (_lib.gemm_workspace_bytes(M, D, F, 0),), u8)}
    if not all(_w.scratch_covers(role, shape, dtype, dev) for role, shape, dtype in roles.values()):
        return None
    bufs = {n: _w.scratch(role, shape, dtype, dev) for n, (role, shape, dtype) in roles.items()}
    args = _lib.EncoderLayers(
        sequences=sequences, rows=rows, final_layer=L - 1, layer_stride=K.shape[-2] * hd, sequence_stride=L * K.shape[-2] * hd if sequences > 1 else 0,
        k_cache=K.data_ptr(), v_cache=V.data_ptr(), row_sums=bufs["sums"].data_ptr(), **{n: t.data_ptr() for n, (t, _) in plain.items()},
        **{n: stacks[s].data_ptr() for n, s in (("qkv_w", "attn_qkv_w"), ("o_w", "attn_o_w"), ("gate_w", "ffn_gate_w"), ("up_w", "ffn_up_w"), ("down_w", "ffn_down_w"))},
        **{f"ws_{n}": bufs[n].data_ptr() for n in ("attn", "o", "down")}, **{f"ws_{n}_bytes": bufs[n].numel() for n in ("attn", "o", "down")})
    if not _lib.offered("fvla_encoder_layers_run", ctypes.byref(args), _w._stream()):      # no layers yet: only whether it takes them
        return None

    def run(first, last):
        args.first, args.last = first, last
        _lib.call("fvla_encoder_layers_run", ctypes.byref(args), _w._stream())
    return run


def decoder_batch_layers(weights, caches, buffers, encoder_seq_len, episodes, layers):
    """The layers of one Euler step of a batch of more than 128 rows: a function that enqueues layers [first, last), or None where
    the ops have to be called one by one (fewer rows have cluster kernels of their own; see `vision_tower`)."""
    w, b, K, V = weights, buffers, caches["encoder_K"], caches["encoder_V"]
    x, shadow = b["decoder_x"], b.get("decoder_x_bf16")
    stacks = {n: w[f"decoder_{n}"] for n in ("attn_qkv_w", "attn_o_w", "ffn_gate_w", "ffn_up_w", "ffn_down_w")}
    if not all(isinstance(t, torch.Tensor) for t in (x, shadow, K, V, *stacks.values())) or x.ndim != 2 or K.ndim != 4 or episodes < 2:
        return None
    M, L, S = x.shape[0], stacks["attn_qkv_w"].shape[0], encoder_seq_len
    D, hd = M // episodes, 256
    shapes = {"attn_qkv_w": (L, _WIDTH, _QKV), "attn_o_w": (L, _Q, _WIDTH), "ffn_gate_w": (L, _WIDTH, _FFN), "ffn_up_w": (L, _WIDTH, _FFN), "ffn_down_w": (L, _FFN, _WIDTH)}
    plain = {"q": (b["decoder_q_buf"], (M * _w.DECODER_HEADS, hd)), "hidden": (b["decoder_hidden"], (M, _FFN)), "rope": (b["decoder_rope_weights"], (D, hd)),
             "norm_factor": (b["decoder_norm_factor_buf"], (M,))}
    if M != D * episodes or S < 1 or not 1 <= layers <= L or not _fits(x, (M, _WIDTH), torch.float32) or not _fits(shadow, (M, _WIDTH)):
        return None
    if not all(_fits(t, s) for t, s in plain.values()) or not all(_fits(stacks[n], s) for n, s in shapes.items()):
        return None
    if K.shape[1] < layers or not _fits(K, (episodes, K.shape[1], S + D, hd)) or not _fits(V, K.shape) or not _lib.load().fvla_decoder_batch_supported(episodes, D):
        return None
    ws_bytes = _lib.gemm_workspace_bytes(M, _QKV, _WIDTH, 0)
    attn_bytes = _lib.load().fvla_decoder_attention_workspace_bytes(D * _w.DECODER_HEADS, S + D)
    roles = (("dec_row_sums", (M * (_WIDTH // 32),), torch.float32), ("dec_qkv_ws", (ws_bytes,), torch.uint8), ("dec_attn_ws", (attn_bytes,), torch.uint8))
    # and what the ops take that these layers do not need: a pool warmed up by the stage serves the ops too, should a later pass go op by op
    spare = tuple((f"dec_{n}_ws", (_lib.gemm_workspace_bytes(M, N, Kd, dual),), torch.uint8)
                  for n, N, Kd, dual in (("o", _WIDTH, _Q, 0), ("gate", _FFN, _WIDTH, 1), ("down", _WIDTH, _FFN, 0)))
    if not all(_w.scratch_covers(*r, x.device) for r in roles):
        return None
    sums, ws, ws_attn = (_w.scratch(*r, x.device) for r in roles)
    for role in spare:
        if _w.scratch_covers(*role, x.device):
            _w.scratch(*role, x.device)
    args = _lib.DecoderBatchLayers(
        x=x.data_ptr(), x_shadow=_w._shadow_of(x) or shadow.data_ptr(), k_cache=K.data_ptr(), v_cache=V.data_ptr(), row_sums=sums.data_ptr(),
        ws_qkv=ws.data_ptr(), ws_qkv_bytes=ws_bytes, ws_attn=ws_attn.data_ptr(), ws_attn_bytes=attn_bytes, layer_stride=(S + D) * hd, episode_stride=K.shape[1] * (S + D) * hd, episodes=episodes, tokens=D,
        prefix=S, layers=layers, **{n: t.data_ptr() for n, (t, _) in plain.items()},
        **{n: stacks[s].data_ptr() for n, s in (("qkv_w", "attn_qkv_w"), ("o_w", "attn_o_w"), ("gate_w", "ffn_gate_w"), ("up_w", "ffn_up_w"), ("down_w", "ffn_down_w"))})
    if not _lib.offered("fvla_decoder_batch_layers_run", ctypes.byref(args), _w._stream()):      # no layers yet: only whether it takes them
        return None

    def run(first, last):
        args.first, args.last = first, last
        _lib.call("fvla_decoder_batch_layers_run", ctypes.byref(args), _w._stream())
    return run


def _own(*names):
    return {n: fused_wrappers.FUSED_WRAPPERS.get(n, _w.ALL_WRAPPERS[n]) for n in names}


# the fused table's entries that the native loops issue
decoder_steps.stands_for = _own("decoder_action_in_proj", "decoder_action_mlp", "decoder_norm_qkv_rope", "decoder_attention", "decoder_out_proj_residual",
                                "decoder_norm_gated_ffn", "decoder_ffn_down_residual", "decoder_action_out_proj", "copy_rows")
decoder_batch_layers.stands_for = _own("decoder_norm_qkv_rope", "decoder_attention", "decoder_out_proj_residual", "decoder_norm_gated_ffn",
                                       "decoder_ffn_down_residual")
vision_tower_as_by_op.stands_for = _own("vision_patch_embed", "vision_norm_qkv", "vision_attention", "vision_out_proj_residual", "vision_norm_ffn_up",
                                        "vision_ffn_down_residual")
encoder_layers.stands_for = _own("encoder_norm_qkv_rope", "encoder_attention", "encoder_out_proj_residual", "encoder_norm_gated_ffn",
                                 "encoder_ffn_down_residual")

STAGES = {"decoder_steps": decoder_steps, "vision_tower": vision_tower_as_by_op, "encoder_layers": encoder_layers,
          "decoder_batch_layers": decoder_batch_layers}
