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


def test_a_layers_numbers_per_head_are_its_own():
    store = KVStore(KVCache(), 1, 2, 64, 1, 64, device="cpu")
    for i in range(20):                                                        # temporaries of one size, as above
        assert float(store._fp32_of(0, "sinks", torch.full((1000,), i, dtype=torch.bfloat16))[0]) == i
    kept = torch.ones(4)
    assert store._fp32_of(0, "gain", kept) is store._fp32_of(0, "gain", kept)


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


def test_rows_that_were_not_selected_for_the_call_are_refused(monkeypatch):
    store, scattered = KVStore(KVCache(), 1, 3, 16, 1, 8, dtype=torch.bfloat16, device="cpu"), []
    monkeypatch.setattr(store, "_scatter", lambda layer, k, v, positions, rows, per_row: scattered.append(rows) or True)
    k, positions = torch.ones(2, 4, 1, 8, dtype=torch.bfloat16), torch.arange(4)[None].repeat(2, 1)
    # the scatter reads one store row per row of the call: other numbers are broadcast or refused by the indexed write
    store.select(torch.tensor([1])).write(0, k, k, positions)
    assert not scattered and bool(store.k[0, 1, :4].all()) and not store.k[0, 0].any()
    with pytest.raises(RuntimeError):
        store.select(torch.tensor([0, 1, 2])).write(0, k, k, positions)
    store.select(torch.tensor([2, 0])).write(0, k, k, positions)
    store.select(None).write(0, k, k, positions)
    assert [None if r is None else r.tolist() for r in scattered] == [[2, 0], None]


class _OnGpu:
    """What the scatter asks a tensor of, as one of a GPU would answer."""

    def __init__(self, shape, device, dtype=torch.bfloat16):
        t = torch.zeros(shape, dtype=dtype)
        self.t, self.device, self.dtype, self.shape, self.is_cuda = t, torch.device(device), dtype, t.shape, True
        self.stride, self.data_ptr, self.numel = t.stride, lambda: 0, t.numel


def test_the_scatter_reads_one_device(monkeypatch):
    store, launched = KVStore(KVCache(), 1, 3, 16, 1, 8, dtype=torch.bfloat16, device="cpu"), []
    monkeypatch.setattr(L, "use_cuda", lambda *t: True)
    monkeypatch.setattr(L, "load", lambda *a: SimpleNamespace(dewb_kv_scatter=lambda *a: launched.append(a)))
    store.k = SimpleNamespace(device=torch.device("cuda:0"))
    k, other, host = _OnGpu((2, 1, 8), "cuda:0"), _OnGpu((2, 1, 8), "cuda:1"), torch.zeros(2, dtype=torch.int32)
    assert not store._scatter(0, k, k, host, None, 1) and not store._scatter(0, k, other, host, None, 1) and not store._scatter(0, other, other, host, None, 1)
    # a warp a token, found by a 32-bit thread number
    positions = SimpleNamespace(numel=lambda: 1 << 27, device=torch.device("cuda:0"), reshape=lambda *s: torch.zeros(1))
    monkeypatch.setattr(L, "status", lambda *a: None)
    monkeypatch.setattr(L, "stream_ptr", lambda: None)
    store.k = store.v = type("Pool", (), {"device": torch.device("cuda:0"), "__getitem__": lambda self, i: None})()
    assert not store._scatter(0, k, k, positions, None, 1)
    assert not launched


def _decoder(**where):
    from dew_b200.models import CausalTransformer
    return CausalTransformer(vocab_size=31, emb_features=32, num_layers=1, num_heads=2, head_dim=16, mlp_features=32, max_seq_len=64, qk_norm=False, **where).eval()


def test_a_prompt_longer_than_its_row_is_refused_on_the_host():
    from dew_b200.sampling.text import RowBatch
    batch, tokens = RowBatch(_decoder(), 2, 16), torch.zeros(2, 20, dtype=torch.long)
    with pytest.raises(ValueError, match="17 tokens"):
        batch.prefill(tokens, torch.tensor([3, 17]))
    assert batch.prefill(tokens, torch.tensor([3, 16])).shape == (2, 31)      # (the padding alone reaches past the rows)


@pytest.mark.gpu
# a position behind the row's last page; a row that the store does not have
@pytest.mark.parametrize("place,row", [(32, 0), (1 << 30, 0), (3, 2)])
def test_what_lies_outside_the_pages_is_reported_and_not_written(place, row):
    store = KVStore(KVCache(page_size=16), 1, 2, 32, 2, 64, device="cuda")
    k = torch.randn(2, 6, 2, 64, generator=torch.Generator().manual_seed(0)).cuda().bfloat16()
    positions = torch.arange(6, device="cuda")[None].repeat(2, 1)
    positions[1] = -1
    positions[1, 5] = place
    rows = torch.tensor([1, row], dtype=torch.int32, device="cuda")
    L.check_status()
    assert store._scatter(0, k[0], k[0], positions, rows, 6)
    with pytest.raises(L.KernelError):
        L.check_status()
    want = torch.zeros_like(store.k)
    want[0, 2, :6] = k[0]
    assert torch.equal(store.k, want) and torch.equal(store.v, want)
