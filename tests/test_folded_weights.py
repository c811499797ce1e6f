"""Where the LayerNorm-folded SigLIP operands are kept and when they are made anew. The library call is replaced by a record of its
arguments: no GPU needed."""
from __future__ import annotations

import pytest
import torch

from flash_vla_b200.hardware.nvidia.b200.pi0.backends.cuda import wrappers

bf16 = torch.bfloat16
K, N, L = 16, 8, 3


@pytest.fixture
def folds(monkeypatch):
    """Destination addresses of the folds so far."""
    made = []

    def call(name, nw, nb, w, b, folded, colsum, bias, n, k, stream):
        assert name == "fvla_fold_layernorm" and n == N and k == K
        made.append((folded, colsum, bias))
    monkeypatch.setattr(wrappers._lib, "call", call)
    monkeypatch.setattr(wrappers, "_chk", lambda name, t, *a, **kw: t.data_ptr())
    monkeypatch.setattr(wrappers, "_stream", lambda: 0)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    return made


def pair(lead=()):
    return [torch.randn(*lead, *s).to(bf16) for s in ((K, N), (K,), (K,), (N,))]


@pytest.mark.parametrize("which", range(4))
def test_refolding_writes_where_captured_graphs_read(folds, which):
    """A graph holds the addresses of the folded operands, not the operands: an update must not give their memory away."""
    single, stacked = pair(), pair((L,))
    first = [wrappers._folded_layernorm(*single)] + wrappers._folded_layers(*stacked)
    held = [tuple(t.data_ptr() for t in f) for f in first]
    assert folds == held
    single[which].mul_(2.0)
    stacked[which].mul_(2.0)
    again = [wrappers._folded_layernorm(*single)] + wrappers._folded_layers(*stacked)
    assert [tuple(t.data_ptr() for t in f) for f in again] == held
    assert folds == held + held
