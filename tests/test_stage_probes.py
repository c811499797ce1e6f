"""The stages' entries say whether they take a plan before they launch anything (first = last = 0: no layers), so that `pipeline` can go
op by op instead: misaligned addresses, pinned plans, kernels switched off, batches that other kernels serve. No GPU needed."""
from __future__ import annotations

import ctypes
import subprocess
import sys

import pytest

from conftest import ROOT

PROBES = """
import ctypes
from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import _lib
lib, P = _lib.load(), 1 << 20
def encoder(sequences=1, rows=768, **change):
    a = _lib.EncoderLayers(sequences=sequences, rows=rows, first=0, last=0, final_layer=17, layer_stride=rows * 256, sequence_stride=18 * rows * 256,
                           **{n: P for n in ("qkv_w", "o_w", "gate_w", "up_w", "down_w", "rope", "x", "x_norm", "q", "attn", "hidden", "k_cache", "v_cache", "row_sums")})
    for n, v in change.items():
        setattr(a, n, v)
    return lib.fvla_encoder_layers_run(ctypes.byref(a), None)
def batch(episodes=5, tokens=51, **change):
    a = _lib.DecoderBatchLayers(episodes=episodes, tokens=tokens, prefix=768, first=0, last=0, layers=18, layer_stride=(768 + tokens) * 256,
                                episode_stride=18 * (768 + tokens) * 256,
                                **{n: P for n in ("qkv_w", "o_w", "gate_w", "up_w", "down_w", "rope", "x", "x_shadow", "q", "hidden", "k_cache", "v_cache", "row_sums")})
    for n, v in change.items():
        setattr(a, n, v)
    return lib.fvla_decoder_batch_layers_run(ctypes.byref(a), None)
def tower(**change):
    a = _lib.VisionTower(views=3, layers=0, **{n: P for n in ("images", "patch_w", "patch_b", "pos_emb", "o_w", "o_b", "down_w", "down_b", "x", "qkv", "attn", "hidden", "row_sums", "ws_patch")})
    for n, v in change.items():
        setattr(a, n, v)
    return lib.fvla_vision_tower_run(ctypes.byref(a), None)
"""


def probe(code, **env):
    import os
    proc = subprocess.run([sys.executable, "-c", PROBES + code], cwd=ROOT, capture_output=True, text=True, env={**os.environ, **env})
    assert proc.returncode == 0, proc.stderr[-800:]


def test_what_the_stages_take_and_refuse():
    probe("""
assert encoder() == 0 and encoder(sequences=8) == 0 and encoder(rows=65) == 0 and encoder(rows=64) == -4
for n in ("x", "attn", "hidden", "k_cache", "gate_w", "row_sums"):
    assert encoder(**{n: P + 2}) == -4 and encoder(**{n: None}) == -4
assert encoder(layer_stride=768 * 256 + 4) == -4 and encoder(layer_stride=256) == -1 and encoder(last=18) == -1 and encoder(rows=0) == -1
assert batch() == 0 and batch(episodes=2, tokens=65) == 0 and batch(episodes=2) == -4 and batch(episodes=2, tokens=129) == -4 and batch(episodes=1, tokens=200) == -4
for n in ("x", "x_shadow", "k_cache", "down_w"):
    assert batch(**{n: P + 2}) == -4 and batch(**{n: None}) == -4
assert tower(x=P + 2) == -4 and tower(ws_patch=P + 8) == -4 and tower(views=0) == -1
assert lib.fvla_row_sums_supported(64) == 0 and lib.fvla_row_sums_supported(65) == 1
assert lib.fvla_gemm_plan_set(768, 2048, 2048, 0, 1, 128, 1) == 0
assert encoder() == -4 and batch() == -4 and tower() == -4 and lib.fvla_row_sums_supported(768) == 0
lib.fvla_gemm_plan_clear()
assert encoder() == 0
""")


@pytest.mark.parametrize("env,one,several", [({"FVLA_GEMM": "mma"}, -4, -4), ({"FVLA_ATTN": "mma"}, 0, -4)])
def test_kernels_switched_off(env, one, several):
    probe(f"assert encoder() == {one} and encoder(sequences=2) == {several}", **env)


LAYERS = """
def arrays(layers=2, **change):
    f = {n: (ctypes.c_void_p * layers)(*([P] * layers)) for n in ("qkv_folded", "qkv_colsum", "qkv_bias", "up_folded", "up_colsum", "up_bias")}
    f.update(change)
    return dict(layers=layers, **{n: a if a is None else ctypes.addressof(a) for n, a in f.items()}), f
"""


def test_tower_refuses_null_pointers():
    """As the other two stages do: before anything is launched, let alone read through the pointer."""
    probe(LAYERS + """
given, keep = arrays()
for n in ("images", "patch_w", "patch_b", "pos_emb", "o_w", "o_b", "down_w", "down_b", "x", "qkv", "attn", "hidden", "row_sums", "ws_patch"):
    assert tower(**given, **{n: None}) == -4, n
""")


def test_tower_refuses_null_arrays_and_entries():
    probe(LAYERS + """
for n in ("qkv_folded", "qkv_colsum", "qkv_bias", "up_folded", "up_colsum", "up_bias"):
    for broken in ((ctypes.c_void_p * 2)(P, None), None):
        given, keep = arrays(**{n: broken})
        assert tower(**given) == -4, n
""")
