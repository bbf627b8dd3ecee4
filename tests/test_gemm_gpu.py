"""Split reductions, wide epilogues with a bias, and column sums, at the edges of their tiles."""
import pytest
import torch

from dew_b200 import ops
from dew_b200.ops import functional as Fn
from dew_b200.ops import library as L

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


def rel_err(a, b):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


# 24 to 74 output tiles with reductions that end inside a step, a part and a whole part; every layout and epilogue
@pytest.mark.parametrize("M,N,K", [(768, 1024, 2048), (1000, 776, 2056), (2304, 768, 4104), (3072, 768, 16384)])
@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
def test_split_reductions(M, N, K, layout):
    assert Fn.reduction_splits(M, N, K) > 1
    g = torch.Generator(device=DEV).manual_seed(K)
    a_mn, b_mn = layout == "tn", layout in ("nn", "tn")
    a = torch.randn((K, M) if a_mn else (M, K), generator=g, device=DEV).bfloat16()
    b = torch.randn((K, N) if b_mn else (N, K), generator=g, device=DEV).bfloat16()
    truth = (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double()
    run = lambda **kw: ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn, kernel="sm100_tcgen05", **kw)
    assert rel_err(run(), truth) < 2e-3                                        # one rounding to bf16
    # the tensor core cuts each of a part's per / 16 sums off at 2^-23 of the running total: half of that on average, all towards zero
    limit = -(-K // Fn.reduction_splits(M, N, K) // 16) * 2.0 ** -24 + 1e-6
    assert rel_err(run(out_dtype=torch.float32), truth) < limit
    wide = torch.ones(M, N + 8, device=DEV)                                    # added to rows of a wider tensor, whose rest stays
    run(out=wide[:, :N], accumulate=True)
    assert rel_err(wide[:, :N], truth + 1) < limit and bool((wide[:, N:] == 1).all())
    low = torch.ones(M, N, device=DEV, dtype=torch.bfloat16)
    run(out=low, accumulate=True, alpha=0.5)
    assert rel_err(low, 0.5 * truth + 1) < 2e-3
    assert torch.equal(run(), run())
    L.check_status()


@pytest.mark.parametrize("kernel", ["sm100_tcgen05", "sm100_pair"])
@pytest.mark.parametrize("M,N,K,offset", [(512, 512, 128, 0), (300, 264, 72, 0), (130, 40, 64, 0), (512, 512, 128, 1)])
def test_bias_in_wide_epilogues(kernel, M, N, K, offset):
    """Whole and cut-off chunks of 32 columns; a bias that does not start on 16 bytes."""
    g = torch.Generator(device=DEV).manual_seed(N)
    a, b = (torch.randn(n, K, generator=g, device=DEV).bfloat16() for n in (M, N))
    bias = torch.randn(N + offset, generator=g, device=DEV).bfloat16()[offset:]
    want = a.double() @ b.double().t() + bias.double()
    assert rel_err(ops.gemm(a, b, bias=bias, kernel=kernel), want) < 2e-3
    L.check_status()


@pytest.mark.parametrize("rows,d", [(256, 8), (257, 264), (1000, 768), (16384, 2304)])
def test_column_sums(rows, d):
    g = torch.Generator(device=DEV).manual_seed(d)
    x = torch.randn(rows, d + 8, generator=g, device=DEV).bfloat16()[:, :d]
    want = x.double().sum(0)
    # fp32 sums, one rounding to bf16 of each
    assert float((Fn._column_sums(x).double() - want).abs().max()) <= float(want.abs().max()) * 2.0 ** -8
    assert rel_err(Fn._column_sums(x), want) < 3e-3
