"""Which small products the few-row kernel is given: on the CPU, with the kernel's launcher replaced by a list of its calls."""
import contextlib
from types import SimpleNamespace

import pytest
import torch

from dew_b200.ops import functional as Fn
from dew_b200.ops import library as L


@pytest.fixture
def launched(monkeypatch):
    calls = []
    monkeypatch.setattr(L, "use_cuda", lambda *t: True)
    monkeypatch.setattr(L, "load", lambda *a: SimpleNamespace(dewb_gemm_rows_bf16=lambda *a: calls.append(a) or 0))
    monkeypatch.setattr(L, "stream", lambda: 0)
    return calls


def _operands(M=2, N=40, K=64):
    g = torch.Generator().manual_seed(N)
    return [torch.randn(s, generator=g).bfloat16() for s in ((M, K), (N, K), (N,))]


def test_one_bias_per_column_reaches_the_kernel(launched):
    x, w, b = _operands()
    Fn.gemm(x, w, bias=b)
    Fn.gemm(x, w)
    assert len(launched) == 2


# the kernel reads N numbers of the bias, wherever it ends
def test_a_bias_of_another_shape_is_broadcast_or_refused(launched):
    x, w, b = _operands()
    want = (x.float() @ w.float().t())
    for other in (b[:1], b[:40].expand(2, 40).contiguous()):
        got = Fn.gemm(x, w, bias=other)
        assert float((got.float() - want - other.float()).norm() / want.norm()) < 2.0 ** -8
    for wrong in (b[:39], torch.cat([b, b])):
        with pytest.raises(RuntimeError):
            Fn.gemm(x, w, bias=wrong)
    assert not launched


def test_operands_on_another_device_are_left_to_the_library_arm(launched):
    x, w, b = _operands()
    for operands in ((w.to("meta"), None), (w, b.to("meta")), (w.to("meta"), b)):
        with contextlib.suppress(RuntimeError):        # (what it refuses, it refuses on the host)
            Fn.gemm(x, operands[0], bias=operands[1])
    assert not launched

