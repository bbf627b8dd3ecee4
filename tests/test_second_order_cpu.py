"""Gradients that are differentiated again: where a kernel would leave no graph, the plain expressions run."""
from types import SimpleNamespace

import pytest
import torch

from dew_b200.ops import ada
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


FORMS = ["norm", "both", "gate", "both, y unused", "both, h unused"]


def _block(form, x, branch, m):
    shift, scale, gate = m.chunk(3, -1)
    if form == "norm":
        return (ada.ada_norm(x, shift, scale),)
    return (ada.gated_add(x, branch, gate),) if form == "gate" else ada.gated_ada_norm(x, branch, gate, shift, scale)


def _case(B, n, d, device="cpu"):
    g = torch.Generator().manual_seed(d)
    r = lambda *s: torch.randn(*s, generator=g).to(device).bfloat16()
    return [r(B, n, d), r(B, n, d), 0.5 * r(B, 3 * d)], r(B, n, d), r(B, n, d), r(B, n, d)


def _second_order(form, leaves, dy, dh, w):
    """The gradients, and what a function of the first one's gradient is differentiated to."""
    outs = [(o, p) for o, p in zip(_block(form, *leaves), {"norm": [dy], "gate": [dh], "both": [dy, dh], "both, y unused": [None, dh], "both, h unused": [dy, None]}[form])
            if p is not None]
    used = [leaves[0], leaves[2]] if form == "norm" else leaves
    first = torch.autograd.grad([o for o, _ in outs], used, [p for _, p in outs], create_graph=True)
    # (what no second gradient reaches, it reaches in neither form; the last call keeps its graph too, so that on the CPU no kernel is asked for)
    second = torch.autograd.grad(sum((t * t).sum() for t in first) + (first[0] * w).sum(), used, create_graph=not dy.is_cuda, allow_unused=True)
    return first, tuple(torch.zeros_like(u) if t is None else t for t, u in zip(second, used))


@pytest.mark.parametrize("form", FORMS)
def test_the_plain_gradients_of_modulated_norms_are_those_of_the_expressions(form, monkeypatch):
    (x, branch, m), dy, dh, w = _case(2, 3, 16)
    leaves = [t.double().requires_grad_() for t in (x, branch, m)]
    dy, dh, w = dy.double(), dh.double(), w.double()
    want = _second_order(form, leaves, dy, dh, w)

    def forward(x, branch, gate, shift, scale, eps):        # in the kernel's place
        h = x if branch is None else x + gate.unsqueeze(1) * branch
        return None if shift is None else ada.modulate(torch.nn.functional.layer_norm(h, h.shape[-1:], None, None, eps), shift, scale), h, None

    monkeypatch.setattr(ada, "_usable", lambda *t: True)
    monkeypatch.setattr(ada, "_forward", forward)
    got = _second_order(form, leaves, dy, dh, w)
    for a, b in zip(got[0] + got[1], want[0] + want[1]):
        assert torch.allclose(a, b, rtol=1e-9, atol=1e-9)


@pytest.mark.gpu
@pytest.mark.parametrize("form", FORMS)
def test_modulated_norms_are_differentiated_twice(form):
    leaves, dy, dh, w = _case(2, 9, 264, "cuda")
    got, want = (_second_order(form, [t.to(dt).requires_grad_() for t in leaves], *(t.to(dt) for t in (dy, dh, w))) for dt in (torch.bfloat16, torch.float64))
    L.check_status()
    # a rounding of h, of each first gradient and of each second one, which reads both
    for a, b in zip(got[0] + got[1], want[0] + want[1]):
        assert float((a.double() - b).norm()) <= 2e-2 * float(b.norm())                  # (both are zero where nothing is reached)
