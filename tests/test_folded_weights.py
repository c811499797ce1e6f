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
    on[0] = 0

    def call(name, nw, nb, w, b, folded, colsum, bias, n, k, stream):
        assert name == "fvla_fold_layernorm" and n == N and k == K
        made.append((folded, colsum, bias))
    monkeypatch.setattr(wrappers._lib, "call", call)
    monkeypatch.setattr(wrappers, "_chk", lambda name, t, *a, **kw: t.data_ptr())
    monkeypatch.setattr(wrappers, "_stream", lambda: on[0])
    monkeypatch.setattr(wrappers, "_fold_recorded", lambda: Done(), raising=False)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    return made


on = [0]                     # the current stream


class Done:
    """Stands for the event behind a fold. (No `query`: a capture in another thread forbids that.)"""
    waits = 0

    def wait(self):
        Done.waits += 1


@pytest.fixture
def folds(monkeypatch):
    """Destination addresses of the folds so far."""
    made = []
    on[0] = 0

    def call(name, nw, nb, w, b, folded, colsum, bias, n, k, stream):
        assert name == "fvla_fold_layernorm" and n == N and k == K
        made.append((folded, colsum, bias))
    monkeypatch.setattr(wrappers._lib, "call", call)
    monkeypatch.setattr(wrappers, "_chk", lambda name, t, *a, **kw: t.data_ptr())
    monkeypatch.setattr(wrappers, "_stream", lambda: on[0])
    monkeypatch.setattr(wrappers, "_fold_recorded", lambda: Done(), raising=False)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    return made


on = [0]                     # the current stream


class Done:
    """Stands for the event behind a fold."""
    reached, waits = False, 0

    def query(self):
        return Done.reached

    def wait(self):
        Done.waits += 1


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


def test_a_norm_in_memory_that_an_earlier_one_had_is_folded(folds):
    """Entries are not found by address: a tensor that took over a freed one's memory, at the same version, is another tensor."""
    arena = torch.empty(1 << 16, dtype=torch.uint8)

    def at(offset, value):                                   # a tensor of its own storage at a given address
        import ctypes
        t = torch.frombuffer((ctypes.c_char * (2 * K)).from_address(arena.data_ptr() + offset), dtype=bf16)
        arena[offset:offset + 2 * K].view(bf16).fill_(value)
        return t
    w, _, nb, b = pair()
    first = at(0, 1.0)
    wrappers._folded_layernorm(w, first, nb, b)
    wrappers._folded_layernorm(w, first, nb, b)
    assert len(folds) == 1
    address, version = first.data_ptr(), first._version
    del first
    second = at(0, 2.0)
    assert (second.data_ptr(), second._version) == (address, version)
    wrappers._folded_layernorm(w, second, nb, b)
    assert len(folds) == 2


def test_folds_of_norms_that_are_gone_are_given_back(folds):
    w, _, nb, b = pair()
    for _ in range(5):
        wrappers._folded_layernorm(w, torch.randn(K).to(bf16), nb, b)
    assert len(getattr(w, wrappers._FOLDED_ATTR)) == 1


def test_folds_are_found_through_views_of_one_storage(folds):
    """Slices made anew on every call, a stack's layers and its own slices, and `data` are the same weights."""
    stacks = pair((L,))
    first = wrappers._folded_layers(*stacks)
    for l in range(L):
        assert wrappers._folded_layernorm(*(t[l] for t in stacks)) is first[l]
    assert all(a is f for a, f in zip(wrappers._folded_layers(*stacks), first)) and len(folds) == L


@pytest.mark.parametrize("stacked", [False, True])
def test_another_stream_waits_for_the_fold(folds, monkeypatch, stacked):
    """Engines that run their episodes on streams of their own fold on the first one's: the others must not read before that has run."""
    sources = pair((L,)) if stacked else pair()
    find, count = (wrappers._folded_layers, L) if stacked else (wrappers._folded_layernorm, 1)
    monkeypatch.setattr(Done, "waits", 0)
    find(*sources)
    find(*sources)
    assert Done.waits == 0                                   # the same stream is in order anyway
    for stream in (1, 2):
        on[0], before = stream, Done.waits
        find(*sources)
        assert Done.waits == before + count
        find(*sources)
        assert Done.waits == before + count                  # and from then on
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    on[0] = 3
    find(*sources)
    assert Done.waits == 2 * count and len(folds) == count
