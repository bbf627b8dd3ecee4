"""The paged cache: the integers of a decode step."""
import pytest
import torch

from dew_b200.nn.kv_cache import KVCache, KVStore


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
