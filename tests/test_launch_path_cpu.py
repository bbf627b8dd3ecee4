"""What lets a call leave out its autograd node, and the environment as every call reads it."""
import os

import pytest
import torch
import torch.autograd.forward_ad as fwd

from dew_b200.ops import library as L


def test_only_calls_that_nothing_records_leave_out_their_node():
    x, w = torch.ones(2), torch.ones(2, requires_grad=True)
    assert L.unrecorded(x) and L.unrecorded(x, None) and not L.unrecorded(x, w)
    with torch.no_grad():
        assert L.unrecorded(x, w)
        with fwd.dual_level():
            assert not L.unrecorded(x)
        seen = []
        torch.func.vmap(lambda t: (seen.append(L.unrecorded(t)), t)[1])(x)
        torch.func.grad(lambda t: (seen.append(L.unrecorded(t)), t.sum())[1])(x)
        torch.jit.trace(lambda t: (seen.append(L.unrecorded(t)), t * 2)[1], (x,), check_trace=False)
        assert seen == [False] * 3
        assert L.unrecorded(x)


def test_environment_is_read_as_it_is_now(monkeypatch):
    monkeypatch.delenv("DEWB_SOME_SWITCH", raising=False)
    assert L.env("DEWB_SOME_SWITCH") is None and L.env("DEWB_SOME_SWITCH", "7") == "7"
    monkeypatch.setenv("DEWB_SOME_SWITCH", "1")
    assert L.env("DEWB_SOME_SWITCH") == os.environ["DEWB_SOME_SWITCH"] == "1"


@pytest.mark.gpu
# one to four rows take the few-row kernel up to its line (2 and 6 M weights), K's pieces short of and past its unrolled steps
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (1, 1, 264), (2, 37, 1032), (3, 2400, 256), (4, 4096, 512), (4, 4104, 512), (1, 6144, 1024), (2, 6152, 1024), (5, 40, 24),
                                   (128, 256, 64)])
def test_small_products_with_and_without_a_node(M, N, K):
    from dew_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w, b = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((M, K), (N, K), (N,)))
    truth = x.double() @ w.double().t() + b.double()
    with torch.no_grad():
        plain = ops.linear(x, w, b)
    recorded = ops.linear(x, w.clone().requires_grad_(), b)
    assert torch.equal(plain, recorded)
    # one rounding of an fp32 sum to bf16: half a unit of eight bits at the most, where a single value is the whole result
    assert float((plain.double() - truth).norm() / truth.norm()) < 2.0 ** -8
    want = x.double() @ w.double().t()
    wide = torch.randn(M, K + 16, generator=g, device="cuda").bfloat16()[:, 8:K + 8]          # rows of a wider tensor
    for a, t in ((x, want), (wide, wide.double() @ w.double().t())):
        assert float((ops.gemm(a, w).double() - t).norm() / t.norm()) < 2.0 ** -8
