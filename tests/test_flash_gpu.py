"""The flash attention kernels at the places where their pipelines can go wrong, against the fp32 reference."""
import pytest
import torch

from dew_b200 import ops
from dew_b200.ops import library as L

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


def rel_err(a, b):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm().clamp_min(1e-12))


@pytest.mark.parametrize("S,docs,seed", [(2048, 6, 0), (2048, 6, 1), (4096, 9, 2), (4096, 40, 3)])
def test_flash_packed_documents_of_uneven_work(S, docs, seed):
    """Documents cut at arbitrary places: the warps of a query tile have unequal work (some rows of a key tile are masked element by element, some rescale,
    some do neither), so fast ones run a tile ahead of slow ones.  bf16 results of fp32 sums: a rounding of the probabilities (2^-9) and one of the result."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    B, Hq, Hkv, D = 2, 8, 2, 128
    # scores that grow along the row make the running maximum move, as trained attention does
    grow = torch.linspace(0.5, 4.0, S, device=DEV)[None, :, None, None]
    q, k, v = (torch.randn(B, S, h, D, generator=g, device=DEV) for h in (Hq, Hkv, Hkv))
    q, k, v = q.bfloat16(), (k * grow).bfloat16(), v.bfloat16()
    seg = torch.ones(B, S, dtype=torch.int32)
    r = torch.Generator().manual_seed(seed)
    for row in seg:
        for cut in (torch.randperm(S - 1, generator=r)[: docs - 1] + 1).tolist():
            row[cut:] += 1
    seg = seg.to(DEV)
    out = ops.attention(q, k, v, segment_ids=seg, kernel="sm100_flash")
    L.check_status()
    assert all(torch.equal(out, ops.attention(q, k, v, segment_ids=seg, kernel="sm100_flash")) for _ in range(5))
    assert rel_err(out, ops.attention_reference(q.float(), k.float(), v.float(), segment_ids=seg)) < 6e-3
