"""A scratch pool that the native stages filled serves the ops they stand for as well: warmed up, frozen, and then a launch plan is pinned, which
sends the pass op by op."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
bf16 = torch.bfloat16


@pytest.mark.parametrize("views,episodes", [(1, 1), (1, 3), (3, 3)])
def test_frozen_pool_serves_the_ops_behind_the_stages(views, episodes):
    from flash_vla_b200 import op_table, random_checkpoint
    from flash_vla_b200.hardware.nvidia.b200.pi0 import pipeline
    from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import _lib, wrappers
    from flash_vla_b200.hardware.nvidia.b200.pi0.buffers import allocate_batched_buffers, allocate_batched_decoder_buffers, allocate_static_buffers
    from flash_vla_b200.runtime.cuda import ScratchPool
    chunk = 50
    w, ops, pool = random_checkpoint(prompt_len=0, wscale=0.02, seed=0, device="cuda"), op_table(), ScratchPool()
    gen = torch.Generator(device="cuda").manual_seed(views)
    if episodes == 1:
        p, S = allocate_static_buffers(views, chunk, 0, "cuda")
        wrappers.register_bf16_shadow(p["decoder_x"], p["decoder_x_bf16"])
    else:
        p, _, S = allocate_batched_buffers(views, chunk, 0, episodes, "cuda")
        d = allocate_batched_decoder_buffers(chunk, episodes, S, "cuda")
    p["observation_images_normalized"].copy_(torch.rand(p["observation_images_normalized"].shape, device="cuda", generator=gen) * 2 - 1)

    def run():
        with wrappers.use_pool(pool):
            pipeline.vision_encoder(ops, w, p, views)
            if episodes == 1:
                pipeline.transformer_encoder(ops, w, p, S)
                p["diffusion_noise"].fill_(0.5)
                pipeline.transformer_decoder(ops, w, p, S, steps=1)
                return p["encoder_K"].clone(), p["diffusion_noise"].clone()
            pipeline.transformer_encoder_batched(ops, w, p, S, views, episodes)
            d["diffusion_noise_f32"].fill_(0.5)
            pipeline.decoder_step_batched(ops, w, {n: p[n] for n in ("encoder_K", "encoder_V")}, d, S, 0, episodes)
            return p["encoder_K"].clone(), d["diffusion_noise_f32"].clone()

    native = run()
    pool.freeze()
    _lib.call("fvla_gemm_plan_set", 777, 2048, 2048, 0, 1, 128, 1)
    try:
        by_op = run()
    finally:
        _lib.call("fvla_gemm_plan_clear")
    for a, b in zip(native, by_op):
        # (a pass of 45 layers and one step: the two op tables are 1.7e-2 apart, by roundings)
        assert torch.isfinite(b).all() and ((a.double() - b.double()).norm() / a.double().norm()).item() <= 3e-2
