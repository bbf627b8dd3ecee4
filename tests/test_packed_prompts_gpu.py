"""Prompts behind one another without their padding: the attention kernel over rows, the cache write, and a model's prefill against the padded form."""
import math

import pytest
import torch

from dew_b200 import ops
from dew_b200.models import CausalTransformer
from dew_b200.nn.kv_cache import KVCache, KVStore, PackedRows
from dew_b200.ops import library as L
from dew_b200.ops.flash import Variants, flash_fwd_rows
from dew_b200.sampling.text import RowBatch, generate

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


def rel_err(a, b):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kind", ["plain", "window", "softcap", "sinks"])
def test_attention_of_rows_behind_one_another(D, kind):
    g = torch.Generator(device=DEV).manual_seed(D)
    tiles, Hq, Hkv = [1, 3, 1, 2, 7], 4, 2
    S = 128 * sum(tiles)
    qkv = torch.randn(S, Hq + 2 * Hkv, D, generator=g, device=DEV).bfloat16()
    q, k, v = qkv[:, :Hq], qkv[:, Hq:Hq + Hkv], qkv[:, Hq + Hkv:]
    first = torch.tensor([sum(tiles[:i]) for i, n in enumerate(tiles) for _ in range(n)], dtype=torch.int32, device=DEV)
    kw = {"plain": {}, "window": dict(window=200), "softcap": dict(softcap=5.0), "sinks": dict(sinks=torch.randn(Hq, generator=g, device=DEV))}[kind]
    out = flash_fwd_rows(q, k, v, D ** -0.5, first, Variants(kw.get("window"), kw.get("softcap", 0.0), kw.get("sinks")))
    L.check_status()
    at = 0
    for n in tiles:
        sl = slice(128 * at, 128 * (at + n))
        want = ops.attention_reference(*(t[sl].float()[None] for t in (q, k, v)), **kw)[0]
        assert rel_err(out[sl], want) < 5e-3                                  # a rounding of the probabilities and one of the result
        at += n


def test_scattered_keys_and_values_lie_where_the_indexed_write_puts_them():
    g = torch.Generator(device=DEV).manual_seed(0)
    R, S, H, D = 3, 70, 2, 64
    qkv = torch.randn(R, S, 2 + 2 * H, D, generator=g, device=DEV).bfloat16()
    pos = torch.arange(S, device=DEV)[None].repeat(R, 1) + 30
    pos[1, 40:] = -1
    stores = [KVStore(KVCache(page_size=16), 2, 5, 128, H, D, device=DEV) for _ in range(2)]
    for s, k, v in zip(stores, (qkv[:, :, 2:2 + H], qkv[:, :, 2:2 + H].contiguous().transpose(0, 1).contiguous().transpose(0, 1)),
                       (qkv[:, :, 2 + H:], qkv[:, :, 2 + H:])):                # (tokens that are not one after another take the indexed write)
        s.page_table.copy_(torch.randperm(s.pages, generator=torch.Generator().manual_seed(1)).reshape(s.rows, -1).int())
        s.select(torch.tensor([4, 0, 2], device=DEV))
        s.write(1, k, v, pos)
    a, b = stores
    assert torch.equal(a.k[:, :a.pages], b.k[:, :b.pages]) and torch.equal(a.v[:, :a.pages], b.v[:, :b.pages]) and bool(a.k.any())


@pytest.mark.parametrize("lengths,extra", [([1, 300, 128, 129, 511], {}), ([200, 20, 20], dict(window=64, num_kv_heads=4)), ([384, 5, 6, 250], dict(qk_norm=True, attention_sinks=True))])
def test_prefill_equals_the_padded_form(lengths, extra, monkeypatch):
    fields = {**dict(vocab_size=97, emb_features=128, num_layers=3, num_heads=4, num_kv_heads=2, head_dim=64, mlp_features=256, max_seq_len=700, qk_norm=False), **extra}
    torch.manual_seed(len(lengths))
    model = CausalTransformer(dtype=torch.bfloat16, device=DEV, **fields).eval()
    R, S = len(lengths), max(lengths)
    tokens, count = torch.randint(0, 97, (R, S), device=DEV), torch.tensor(lengths, device=DEV)
    batches, out = [], []
    for packed in (True, False):
        if not packed:
            monkeypatch.setenv("DEWB_KERNEL_ATTENTION", "sm100_flash" if S % 128 == 0 else "sdpa")
        b = RowBatch(model, R, 640, kv_cache=KVCache(page_size=64))
        assert PackedRows.takes(b.store, model, lengths, S) == packed
        first = b.prefill(tokens, count)
        monkeypatch.delenv("DEWB_KERNEL_ATTENTION", raising=False)
        batches.append(b)
        out.append((first, b.forward(tokens[:, :1], count[:, None])[:, 0]))
    L.check_status()
    for a, b in zip(*out):
        assert rel_err(a, b) < 2e-2                                            # bf16 through three layers, two attention kernels
    (sa, sb) = (b.store for b in batches)
    live = torch.zeros(R, sa.max_pages * 64, dtype=torch.bool, device=DEV)
    for r, n in enumerate(lengths):
        live[r, :n + 1] = True
    for a, b in ((sa.k, sb.k), (sa.v, sb.v)):
        a, b = (t[:, :sa.pages].reshape(3, R, -1, *t.shape[3:]) for t in (a, b))
        assert rel_err(a[:, live], b[:, live]) < 2e-2 and not bool(a[:, ~live].any()) and math.isfinite(float(a.float().sum()))


def test_generation_from_prompts_of_uneven_lengths():
    torch.manual_seed(0)
    model = CausalTransformer(dtype=torch.bfloat16, device=DEV, vocab_size=97, emb_features=128, num_layers=2, num_heads=2, head_dim=64, mlp_features=256, max_seq_len=400,
                              qk_norm=False).eval()
    prompts = [torch.randint(0, 97, (n,)).tolist() for n in (3, 300, 150)]
    out = generate(model, None, prompts, 4)
    assert out.prompt_lengths.tolist() == [3, 300, 150] and out.tokens.shape == (3, 304)
    L.check_status()
