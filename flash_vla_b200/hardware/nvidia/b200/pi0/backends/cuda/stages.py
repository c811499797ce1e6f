"""Whole stages of the pipeline as one call into the library.

Not call sites of the reference's op table: `op_table(fused=True)` carries them beside the ops. A stage names the ops it
stands for (`stands_for`); `pipeline` takes it while the table still has exactly those, else it issues the table's own ops one by one.
"""
from __future__ import annotations

import ctypes

import torch

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


# the fused table's entries that the native loop issues
decoder_steps.stands_for = {n: fused_wrappers.FUSED_WRAPPERS.get(n, _w.ALL_WRAPPERS[n]) for n in (
    "decoder_action_in_proj", "decoder_action_mlp", "decoder_norm_qkv_rope", "decoder_attention", "decoder_out_proj_residual",
    "decoder_norm_gated_ffn", "decoder_ffn_down_residual", "decoder_action_out_proj", "copy_rows")}

STAGES = {"decoder_steps": decoder_steps}
