"""Gradients that are differentiated again: where a kernel would leave no graph, the plain expressions run."""
from types import SimpleNamespace

import torch

from dew_b200.ops import functional as Fn
from dew_b200.ops import library as L


def test_a_bias_gradient_keeps_its_graph(monkeypatch):
    launched = []

    class Lib(SimpleNamespace):
        def __getattr__(self, name):
            return lambda *a: launched.append(name) or 1

    monkeypatch.setattr(L, "use_cuda", lambda *t: True)
    monkeypatch.setattr(L, "load", lambda *a: Lib())
    monkeypatch.setattr(L, "stream_ptr", lambda: None)
    monkeypatch.setattr(L, "check", lambda *a: None)
    dy = torch.randn(256, 8).bfloat16().requires_grad_()
    db = Fn._column_sums(dy)
    assert not launched and torch.equal(torch.autograd.grad(db.sum(), dy)[0], torch.ones_like(dy))
    with torch.no_grad():                              # (an ordinary backward)
        Fn._column_sums(dy)
    Fn._column_sums(dy.detach())
    assert launched.count("dewb_colsum_bf16") == 2
