"""Which small products the few-row kernel is given: on the CPU, with the kernel's launcher replaced by a list of its calls."""
import contextlib
import os
import subprocess
import sys
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


# the library arm keeps what it does faster: long reductions (it splits them), many columns of short ones, more than a few megabytes
@pytest.mark.parametrize("M,N,K", [(1, 8, 262144), (2, 64, 16384), (1, 384, 8192), (4, 512, 2048), (3, 256, 4096), (2, 65536, 16), (2, 8192, 128), (4, 8192, 256), (1, 32000, 1024), (5, 8, 8)])
def test_products_that_the_library_arm_does_faster_stay_there(launched, M, N, K):
    assert not Fn._few_rows(M, N, K)


def test_the_few_row_kernel_keeps_what_it_does_faster():
    assert all(Fn._few_rows(*s) for s in [(1, 8, 8), (1, 2048, 1024), (2, 3072, 2048), (1, 12288, 512), (2, 64, 8192), (4, 32, 8192), (4, 2048, 1024), (3, 4096, 256), (2, 1536, 4096)])


def test_the_measured_cell_is_the_kernels_own(launched, monkeypatch):
    from dew_b200.ops.selection import route_report
    x, w, b = _operands()
    route_report(reset=True)
    Fn.gemm(x, w, bias=b)
    assert route_report()["gemm"] == {"sm100_rows": {"calls": 1, "forced": 0, "declared_cell": 1, "after_refusals": {}}}
    # an explicit DEWB_DECODE_GEMM leaves no cell of the few-row kernel, and its entry refuses what the library arm does faster
    monkeypatch.delitem(Fn._GEMM.declared, ("rows",))
    Fn.gemm(x, w, bias=b)
    assert len(launched) == 1
    entry = next(k for k in Fn._GEMM.kernels if k.name == "sm100_rows")
    case = dict(M=2, K=64, lda=64, ldb=64, ldd=40, aligned=True, inner_contig=True, dtype=torch.bfloat16, plain=True, k_major=True, row_operands=True)
    assert not entry.refusals(dict(case, N=36)) and entry.refusals(dict(case, N=36004)) and entry.refusals(dict(case, N=36, row_operands=False))


def test_an_explicit_choice_of_the_decode_kernel_holds_for_few_rows():
    code = "from dew_b200.ops import functional as F; print(sorted(F._GEMM.declared.items()))"
    out = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, DEWB_DECODE_GEMM="cublas"), capture_output=True, text=True, check=True,
                         cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__)))).stdout
    assert "('decode',), 'cublas'" in out and "rows" not in out


@pytest.mark.gpu
# one, two and four columns a warp, at the last and first sizes of each; the longest reduction; three and four rows
@pytest.mark.parametrize("M,N,K", [(1, 4735, 256), (2, 4736, 264), (1, 9471, 256), (2, 9473, 264), (2, 12288, 512), (2, 9, 8192), (3, 4095, 256), (4, 31, 8192)])
def test_few_rows_against_64_bits(M, N, K):
    from dew_b200.ops.selection import route_report
    x, w, b = (t.cuda() for t in _operands(M, N, K))
    if N >= 6144:                                      # (with a bias the dense kernel's epilogue takes them)
        b = None
    route_report(reset=True)
    y = Fn.gemm(x, w, bias=b)
    assert route_report()["gemm"]["sm100_rows"]["calls"] == 1
    want = x.double() @ w.double().t() + (0 if b is None else b.double())
    assert float((y.double() - want).norm() / want.norm()) < 2.0 ** -8                # one rounding of an fp32 sum to bf16
