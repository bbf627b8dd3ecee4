"""The activation of a diffusion transformer's condition: one for all that are given it, and none where nobody is."""
import pytest
import torch
import torch.nn.functional as F

from dew_b200.models import SimpleDiT


@pytest.mark.parametrize("adaln_silu,watched,made", [(True, (), 1), (True, (0, 1, 2), 3), (True, (0, 1), 3), (False, (), 1), (False, (2,), 1)])
def test_the_condition_is_activated_as_often_as_needed(adaln_silu, watched, made, monkeypatch):
    torch.manual_seed(0)
    model = SimpleDiT(patch_size=4, emb_features=32, num_layers=2, num_heads=2, adaln_silu=adaln_silu)
    for p in model.parameters():
        torch.nn.init.normal_(p, std=0.1)
    x, t = torch.randn(3, 8, 8, 3), torch.rand(3)
    plain = model(x, t)
    condition, silu = [], F.silu
    model.conditioning.register_forward_hook(lambda m, args, out: condition.append(out))
    for i in watched:
        (*model.blocks, model.output)[i].register_forward_hook(lambda *a: None)
    calls = []
    monkeypatch.setattr(F, "silu", lambda v, *a, **k: (calls.append(any(v is c for c in condition)), silu(v, *a, **k))[1])
    assert torch.equal(model(x, t), plain)
    assert sum(calls) == made
