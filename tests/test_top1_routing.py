"""One expert a token: the routing weight's gradient, with weights that depend on the scores and with weights that do not."""
from types import SimpleNamespace

import pytest
import torch

from dew_b200.models.causal_transformer import Mixture
from dew_b200.nn import moe as M
from dew_b200.ops import library as L
from dew_b200.parallel import ep


def test_which_weights_do_not_depend_on_the_scores():
    mix = lambda **kw: Mixture(experts=4, **kw)
    assert ep.constant_weights(mix(top_k=1, norm_topk_prob=True)) and ep.constant_weights(mix(top_k=1, norm_topk_prob=False, score_function="top_softmax"))
    assert not ep.constant_weights(mix(top_k=1, norm_topk_prob=False)) and not ep.constant_weights(mix(top_k=2, norm_topk_prob=True))


@pytest.mark.parametrize("k", [1, 3])
def test_a_weight_that_depends_on_the_scores_takes_the_kernel(monkeypatch, k):
    launched = []
    monkeypatch.setattr(L, "load", lambda *a: SimpleNamespace(dewb_moe_pair_dots=lambda *a: launched.append(a) or 0))
    monkeypatch.setattr(L, "stream_ptr", lambda: None)
    rows, dy = torch.randn(5 * k, 16), torch.randn(5, 16)
    ctx = SimpleNamespace(saved_tensors=(torch.rand(5, k), rows), plan=SimpleNamespace(tokens=5, top_k=k), exchange=SimpleNamespace(push=lambda *a, **kw: None), constant=False)
    ep._PullRows.backward(ctx, dy)
    assert len(launched) == 1
    ctx.constant = True
    dw = ep._PullRows.backward(ctx, dy)[1]
    assert len(launched) == 1 and torch.allclose(dw, (rows.view(5, k, 16) * dy[:, None]).sum(-1))


@pytest.mark.gpu
def test_top1_routing_with_and_without_normalised_weights():
    grads = {}
    for norm in (False, True):
        for kernels in (True, False):
            torch.manual_seed(0)
            layer = M.SparseMLP(256, Mixture(experts=8, top_k=1, expert_features=128, norm_topk_prob=norm), 512).to("cuda", torch.bfloat16)
            layer.use_kernels = kernels
            x = torch.randn(300, 256, device="cuda").bfloat16()
            layer(x).backward(torch.randn(300, 256, device="cuda").bfloat16())
            grads[norm, kernels] = layer.router.weight.grad.double()
    L.check_status()
    real = grads[False, False]
    assert float((grads[False, True] - real).norm()) < 5e-2 * float(real.norm())        # (the two forms round the experts' rows to bf16 at different places)
    # a normalised weight is 1: nothing but rounding reaches the router
    assert all(float(grads[True, kernels].norm()) < 1e-4 * float(real.norm()) for kernels in (True, False))
