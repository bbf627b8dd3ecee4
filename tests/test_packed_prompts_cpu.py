"""Which prefills lay their prompts behind one another: decided on the host, here for a store that says it is on a GPU."""
from types import SimpleNamespace

import pytest
import torch

from dew_b200.models import CausalTransformer
from dew_b200.models.causal_transformer import Mixture
from dew_b200.nn.kv_cache import PackedRows
from dew_b200.ops import library as L

LENGTHS = [1, 300, 128]


@pytest.fixture
def takes(monkeypatch):
    monkeypatch.setattr(L, "load", lambda *a: SimpleNamespace(dewb_flash_fwd_rows=None))
    store = SimpleNamespace(slots=None, kind=0, dtype=torch.bfloat16, device=torch.device("cuda"), row_ids=None, head_dim=64, kv_heads=2, rows=3)
    return lambda model, lengths=LENGTHS, width=300: PackedRows.takes(store, model, lengths, width)


def _decoder(**more):
    fields = dict(vocab_size=31, emb_features=64, num_layers=2, num_heads=2, num_kv_heads=2, head_dim=64, mlp_features=64, max_seq_len=400, qk_norm=False)
    return CausalTransformer(dtype=torch.bfloat16, **{**fields, **more}).eval()


def test_uneven_prompts_of_a_plain_decoder_are_packed(takes):
    model = _decoder()
    assert takes(model) and not takes(model, [300, 299, 290]) and not takes(model, [0, 300, 5]) and not takes(model, [1, 5])


def test_experts_of_several_ranks_keep_the_padded_form(takes):
    model = _decoder(mixture=Mixture(experts=4, top_k=2, expert_features=64))
    assert takes(model)
    for world, packed in ((1, True), (2, False)):
        model.layers[-1].mlp.ep = SimpleNamespace(world=world)
        assert takes(model) == packed


def test_a_watched_decoder_keeps_the_padded_form(takes):
    from dew_b200.nn.inspection import ActivationWatch
    from dew_b200.utils.hooks import moves_weights
    model = _decoder()
    with ActivationWatch(model, ["layers.1.mlp"]):
        assert not takes(model)
    assert takes(model)
    look = lambda *args: None
    for register in (model.register_forward_hook, model.layers[0].mixer.register_forward_pre_hook, torch.nn.modules.module.register_module_forward_hook,
                     torch.nn.modules.module.register_module_forward_pre_hook):
        handle = register(look)
        assert not takes(model)
        handle.remove()
    # a hook that brings a layer's weights sees nothing of its tokens
    model.layers[0].register_forward_pre_hook(moves_weights(lambda *args: None))
    assert takes(model)


def test_lengths_are_read_only_where_they_decide(monkeypatch):
    from dew_b200.sampling.text import RowBatch

    class Lengths(torch.Tensor):
        def tolist(self):
            raise AssertionError("read from the device")

    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    batch = RowBatch(CausalTransformer(vocab_size=31, emb_features=32, num_layers=1, num_heads=2, head_dim=16, mlp_features=32, max_seq_len=200, qk_norm=False).eval(), 2, 200)
    batch.device = torch.device("cuda")                                        # (its store is on the host and its heads are narrow: never packed)
    assert batch.prefill(torch.zeros(2, 150, dtype=torch.long), torch.tensor([3, 150]).as_subclass(Lengths)).shape == (2, 31)
