"""Whole stages of the pipeline as one call into the library.

Not call sites of the reference's op table: `op_table(fused=True)` carries them beside the ops, and `pipeline` takes a
stage when the table has it, else it issues the stage's ops one by one.
"""
from __future__ import annotations

import ctypes

import torch

from . import _lib
from . import wrappers as _w

_WIDTH, _QKV, _Q, _FFN, _ACT = 1024, 2560, 2048, 4096, 32


def decoder_steps(weights, buffers, encoder_seq_len, steps, layers, first_step=0) -> bool:
    """Euler steps [first_step, steps) of the action expert: `pipeline.transformer_decoder` without the state projection,
    the launches of its ops issued from native code. Outside a CUDA graph a step is bound by its 93 calls otherwise:
    18 us each through the op wrappers, on the 51-row call sites that run 5 - 8 us. Returns False, having done nothing,
    for buffers that are not the fp32 residual-stream plan."""
    b, w = buffers, weights
    noise, master, x = b["diffusion_noise"], b.get("diffusion_noise_f32"), b["decoder_x"]
    if master is None or x.dtype != torch.float32 or layers < 1 or tuple(w["decoder_attn_qkv_w"].shape[1:]) != (_WIDTH, _QKV):
        return False
    K, V = b["encoder_K"], b["encoder_V"]
    total, D = w["decoder_attn_qkv_w"].shape[0], x.shape[0]
    if layers > total or K.shape[0] < layers:
        return False
    chunk, rows = D - 1, K.shape[1]
    chk, dev, lib = _w._chk, x.device, _lib.load()

    def scratch(role, M, N, Kd, dual=0):
        return _w._ws(role, _lib.gemm_workspace_bytes(M, N, Kd, dual), dev)

    ws = {"mlp": scratch("dec_mlp_ws", chunk, _WIDTH, _WIDTH), "qkv": scratch("dec_qkv_ws", D, _QKV, _WIDTH),
          "attn": _w._ws("dec_attn_ws", lib.fvla_decoder_attention_workspace_bytes(D * _w.DECODER_HEADS, rows), dev),
          "o": scratch("dec_o_ws", D, _WIDTH, _Q), "gate": scratch("dec_gate_ws", D, _FFN, _WIDTH, 1),
          "down": scratch("dec_down_ws", D, _WIDTH, _FFN)}
    args = _lib.DecoderSteps(
        in_w=chk("in_w", w["decoder_action_fused_in_proj_w"], (_ACT, _WIDTH)),
        time_bias=chk("time_biases", w["decoder_action_fused_time_biases"], (10, _WIDTH)),
        mlp_w=chk("mlp_w", w["decoder_action_mlp_w"], (_WIDTH, _WIDTH)), mlp_b=chk("mlp_b", w["decoder_action_mlp_b"], (_WIDTH,)),
        qkv_w=chk("qkv_w", w["decoder_attn_qkv_w"]), attn_o_w=chk("attn_o_w", w["decoder_attn_o_w"], (total, _Q, _WIDTH)),
        gate_w=chk("gate_w", w["decoder_ffn_gate_w"], (total, _WIDTH, _FFN)), up_w=chk("up_w", w["decoder_ffn_up_w"], (total, _WIDTH, _FFN)),
        down_w=chk("down_w", w["decoder_ffn_down_w"], (total, _FFN, _WIDTH)),
        out_w=chk("out_w", w["decoder_action_fused_out_proj_w"], (_WIDTH, _ACT)), out_b=chk("out_b", w["decoder_action_fused_out_proj_b"], (_ACT,)),
        rope=chk("rope", b["decoder_rope_weights"], (D, 256)), state=chk("state", b["decoder_state_buf"], (1, _WIDTH)),
        noise=chk("noise", noise, (chunk, _ACT)), noise_f32=chk("noise_f32", master, (chunk, _ACT), torch.float32),
        x=chk("decoder_x", x, (D, _WIDTH), torch.float32), x_shadow=_w._shadow_of(x), in_buf=chk("decoder_x_buf", b["decoder_x_buf"], (chunk, _WIDTH)),
        q=chk("decoder_q_buf", b["decoder_q_buf"], (D * _w.DECODER_HEADS, 256)), hidden=chk("decoder_hidden", b["decoder_hidden"], (D, _FFN)),
        k_cache=chk("encoder_K", K, (K.shape[0], encoder_seq_len + D, 256)), v_cache=chk("encoder_V", V, K.shape),
        chunk=chunk, prefix=encoder_seq_len, cache_rows=rows, first_step=first_step, steps=steps, layers=layers,
        **{f"ws_{k}": v[0] for k, v in ws.items()}, **{f"ws_{k}_bytes": v[1] for k, v in ws.items()})
    _lib.call("fvla_decoder_steps_run", ctypes.byref(args), _w._stream())
    return True


STAGES = {"decoder_steps": decoder_steps}
