"""A decoder's layers issued by one call: the same bits as the layers' own way, and only where the layers would do nothing else."""
import pytest
import torch

from dew_b200.models import CausalTransformer, decode_step
from dew_b200.nn.kv_cache import KVCache, KVStore
from dew_b200.sampling.text import RowBatch

DEV = "cuda"


def decoder(device, width=256, heads=4, kv=2, ff=512, layers=3, **kw):
    torch.manual_seed(0)
    return CausalTransformer(vocab_size=128, emb_features=width, num_layers=layers, num_heads=heads, num_kv_heads=kv, head_dim=128, mlp_features=ff, max_seq_len=512, tie_embeddings=False,
                             dtype=torch.bfloat16, device=device, **{"qk_norm": False, **kw}).eval()


def rows_of(model, rows, length=130):
    batch = RowBatch(model, rows, 400, kv_cache=KVCache(page_size=64))
    tokens = torch.randint(0, 128, (rows, length), device=batch.device)
    lengths = torch.full((rows,), length, device=batch.device) - torch.arange(rows, device=batch.device)
    batch.prefill(tokens, lengths)
    return batch, lengths


def test_only_on_the_gpu():
    model = decoder("cpu")
    batch, lengths = rows_of(model, 1)
    h = torch.zeros(1, 1, 256, dtype=torch.bfloat16)
    with torch.no_grad():
        assert decode_step.run(model, h, *model.rope_tables("cpu"), lengths[:, None], batch.store) is None


class Taken:
    """Counts the steps that went as one call."""

    def __init__(self, monkeypatch):
        self.n, run = 0, decode_step.run

        def counted(*a):
            done = run(*a)
            self.n += done is not None
            return done
        monkeypatch.setattr(decode_step, "run", counted)


@pytest.mark.gpu
# one row and the most; one layer (no stream behind a stream) and several; eight heads a key head; windows short of and past the rows, sinks
@pytest.mark.parametrize("rows,kw", [(1, {}), (2, dict(layers=1)), (4, dict(width=128, heads=2, kv=1, ff=264)), (1, dict(heads=8, kv=1, ff=1024)), (2, dict(window=64)),
                                     (1, dict(window=1000, layers=2)), (2, dict(attention_sinks=True))])
def test_same_bits_as_the_layers(rows, kw, monkeypatch):
    model = decoder(DEV, **kw)
    if kw.get("attention_sinks"):
        for layer in model.layers:
            torch.nn.init.normal_(layer.mixer.sinks)
    batch, lengths = rows_of(model, rows)
    ids = torch.randint(0, 128, (rows, 3), device=DEV)
    taken = Taken(monkeypatch)
    one = [batch.forward(ids[:, i:i + 1], (lengths + i)[:, None]).clone() for i in range(3)]
    assert taken.n == 3
    keys, values = batch.store.k.clone(), batch.store.v.clone()
    hook = model.layers[-1].register_forward_hook(lambda *a: None)                # somebody looks on: the layers go one by one
    by_layers = [batch.forward(ids[:, i:i + 1], (lengths + i)[:, None]).clone() for i in range(3)]
    hook.remove()
    assert taken.n == 3
    assert all(torch.equal(a, b) for a, b in zip(one, by_layers))
    assert torch.equal(keys, batch.store.k) and torch.equal(values, batch.store.v)


@pytest.mark.gpu
def test_a_store_knows_its_device(monkeypatch):
    """Asked for on "cuda", it is on the current device, as the rows are."""
    model = decoder(DEV)
    batch, lengths = rows_of(model, 1)
    batch.store = KVStore(KVCache(page_size=64), len(model.layers), 1, 400, 2, 128, torch.bfloat16, "cuda")
    assert batch.store.device == lengths.device
    taken = Taken(monkeypatch)
    batch.forward(torch.zeros(1, 1, dtype=torch.long, device=DEV), torch.zeros(1, 1, dtype=torch.long, device=DEV))
    assert taken.n == 1


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [dict(qk_norm=True), dict(mlp_activation="gelu_tanh"), dict(attn_bias=True), dict(qkv_bias=True), dict(residual_multiplier=0.5), dict(sandwich_norm=True),
                                dict(attn_softcap=30.0), dict(query_scale=0.2), dict(attn_out_gate=True)])
def test_other_layers_go_their_own_way(kw, monkeypatch):
    model = decoder(DEV, **kw)
    batch, lengths = rows_of(model, 1)
    taken = Taken(monkeypatch)
    batch.forward(torch.zeros(1, 1, dtype=torch.long, device=DEV), lengths[:, None])
    assert taken.n == 0


@pytest.mark.gpu
def test_weights_are_looked_at_anew(monkeypatch):
    """A weight that is replaced, or that is no longer in one piece, between two steps."""
    model = decoder(DEV)
    batch, lengths = rows_of(model, 1)
    token = torch.zeros(1, 1, dtype=torch.long, device=DEV)
    taken = Taken(monkeypatch)
    step = lambda: batch.forward(token, lengths[:, None]).clone()
    before = step()
    down = model.layers[1].mlp.down_proj
    down.weight = torch.nn.Parameter(down.weight.detach() * 2)
    changed = step()
    assert taken.n == 2 and not torch.equal(before, changed)
    down.weight = torch.nn.Parameter(down.weight.detach().t().contiguous().t())
    assert torch.allclose(step().float(), changed.float(), rtol=0.05, atol=0.05) and taken.n == 2
    rows = RowBatch(model, 5, 400, kv_cache=KVCache(page_size=64))
    rows.forward(torch.zeros(5, 1, dtype=torch.long, device=DEV), torch.zeros(5, 1, dtype=torch.long, device=DEV))
    assert taken.n == 2
