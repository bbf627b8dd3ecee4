"""The paged cache: the integers of a decode step, and writes of many tokens."""
from types import SimpleNamespace

import pytest
import torch

from dew_b200.nn.kv_cache import KVCache, KVStore
from dew_b200.ops import library as L


def test_a_step_reads_its_own_positions():
    # temporaries of one size: the allocator gives each the address of the one before, which has been freed
    for rows in (64, 1000, 1 << 14):
        store = KVStore(KVCache(), 1, 2, 64, 1, 64, device="cpu")
        for i in range(20):
            pos, lens = store._step_ints(torch.full((rows,), i))
            assert (int(pos[0]), int(lens[-1])) == (i, i + 1)
    # layers of one step pass views of the same positions and share the copies; a change in place makes new ones
    positions = torch.tensor([[3], [-1]])
    first = store._step_ints(positions.reshape(-1))
    assert store._step_ints(positions.reshape(-1))[0] is first[0]
    positions.add_(1)
    assert [t.tolist() for t in store._step_ints(positions.reshape(-1))] == [[4, 0], [5, 1]]


def test_a_decode_step_reads_the_sinks_as_they_are_now(monkeypatch):
    store, seen = KVStore(KVCache(), 1, 2, 64, 1, 64, device="cpu"), []
    monkeypatch.setattr(L, "load", lambda *a: SimpleNamespace(dewb_rope_append=lambda *a: 0))
    monkeypatch.setattr(L, "stream", lambda: 0)
    monkeypatch.setattr(store, "_fused_decode", lambda lib, layer, q, stride, lens, R, Hq, D, window, sinks, out: seen.append(sinks.tolist()))
    sinks = torch.tensor([1.0, 2.0], dtype=torch.bfloat16)
    for _ in range(2):
        store.decode_packed(0, torch.zeros(2, 4, 64), None, None, torch.tensor([0, 1]), 2, sinks=sinks)
        sinks.mul_(2)                                                          # an update of the parameter in place
    assert seen == [[1.0, 2.0], [2.0, 4.0]]


def test_no_rows_write_nothing():
    store = KVStore(KVCache(), 1, 2, 16, 1, 8, device="cpu")
    for S in (0, 3):
        store.write(0, torch.ones(0, S, 1, 8), torch.ones(0, S, 1, 8), torch.zeros(0, S, dtype=torch.long))
    store.write(0, torch.ones(2, 0, 1, 8), torch.ones(2, 0, 1, 8), torch.zeros(2, 0, dtype=torch.long))
    assert not store.k.any()
