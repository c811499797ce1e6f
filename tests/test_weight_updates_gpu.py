"""In-place updates of the weights under engines and graphs that already exist."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
bf16 = torch.bfloat16


# five views: SigLIP QKV folded by the op, FFN up not; six: neither
@pytest.mark.parametrize("views,episodes", [(5, 1), (3, 2)])
def test_captured_batch_follows_updates_of_the_siglip_weights(views, episodes):
    """Beyond four views per replay the op table reads the SigLIP weights themselves: so must a captured engine, or its cache goes stale."""
    from flash_vla_b200 import Pi0Inference, random_checkpoint
    weights = random_checkpoint(prompt_len=0, wscale=0.02, seed=0, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(views)
    lead = (episodes,) if episodes > 1 else ()
    inputs = ((torch.rand(*lead, views, 224, 224, 3, device="cuda", generator=gen) * 2 - 1).to(bf16),
              torch.randn(*lead, 32, device="cuda", generator=gen).to(bf16), torch.randn(*lead, 10, 32, device="cuda", generator=gen).to(bf16))

    def engine():
        return Pi0Inference(weights, num_views=views, chunk_size=10, steps=1, layers=1, episodes=episodes)

    def caches(e):
        e.forward(*inputs)
        return [b[n].clone() for b in e.episode_buffers for n in ("encoder_K", "encoder_V")]

    captured = engine()
    before = caches(captured)
    names = ["ffn_up_w", "ffn_up_b", "pre_ffn_norm_w", "pre_ffn_norm_b"]
    if views * episodes > 5:
        names += ["attn_qkv_w", "attn_qkv_b", "pre_attn_norm_w", "pre_attn_norm_b"]
    for n in names:
        weights["vision_" + n].mul_(1.25).add_(0.01)
    after, fresh = caches(captured), caches(engine())
    for a, b, f in zip(after, before, fresh):
        assert not torch.equal(a, b), "the update does not show"
        assert torch.equal(a, f), "not what an engine captured after the update gives"


def test_refolded_weights_reach_graphs_that_were_captured_before():
    """Up to four views the graph reads folded copies: stale until a pass outside a graph folds again, then current, in the same memory."""
    from flash_vla_b200 import Pi0Inference, random_checkpoint
    weights = random_checkpoint(prompt_len=0, wscale=0.02, seed=0, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(1)
    inputs = ((torch.rand(1, 224, 224, 3, device="cuda", generator=gen) * 2 - 1).to(bf16),
              torch.randn(32, device="cuda", generator=gen).to(bf16), torch.randn(10, 32, device="cuda", generator=gen).to(bf16))

    def engine():
        return Pi0Inference(weights, num_views=1, chunk_size=10, steps=1, layers=1)

    def cache(e):
        e.forward(*inputs)
        return e.buffers["encoder_K"].clone()

    captured = engine()
    before = cache(captured)
    for n in ("attn_qkv_w", "pre_attn_norm_b", "ffn_up_w", "pre_ffn_norm_w"):
        weights["vision_" + n].mul_(1.25).add_(0.01)
    fresh = cache(engine())                                  # its warm-up folds again
    assert not torch.equal(fresh, before)
    assert torch.equal(cache(captured), fresh)
