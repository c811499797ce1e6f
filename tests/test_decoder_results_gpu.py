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


if __name__ == "__main__":
    print(json.dumps({f"projections {M}": projections(M) for M in (1, 33, 51, 64)}, indent=1))
