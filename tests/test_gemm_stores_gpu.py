"""How the products' accumulators reach memory: rows on 32-byte boundaries, rows on 16-byte boundaries only, and columns past the last whole piece."""
import pytest
import torch

from dew_b200 import ops
from dew_b200.ops import library as L
from dew_b200.ops import mx

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


# a row length of 16 (mod 32) bytes puts every second row on a 16-byte boundary; a first column of 8 shifts all; 20 columns past a piece of 32 are stored one by one
@pytest.mark.parametrize("kernel", ["sm100_pair", "sm100_tcgen05"])
@pytest.mark.parametrize("dtype,acc", [(torch.bfloat16, False), (torch.bfloat16, True), (torch.float32, False), (torch.float32, True)])
@pytest.mark.parametrize("N,width,col", [(256, 256, 0), (256, 264, 0), (256, 280, 8), (148, 160, 4), (64, 72, 8)])
def test_rows_of_any_alignment(kernel, dtype, acc, N, width, col):
    if dtype == torch.bfloat16 and col % 8:
        col = 8                                                       # (an output is on a 16-byte boundary)
    g = torch.Generator(device=DEV).manual_seed(N + width + col)
    A, B = (torch.randn(n, 192, generator=g, device=DEV).bfloat16() for n in (300, N))
    held = torch.randn(300, width, generator=g, device=DEV).to(dtype)
    whole = held.clone()
    ops.gemm(A, B, out=whole[:, col:col + N], accumulate=acc, kernel=kernel)
    L.check_status()
    exact = A.double() @ B.double().T + (held[:, col:col + N].double() if acc else 0)
    # fp32 sums of 192 exact products in some order, and one rounding of the result
    bound = 192 * 2.0 ** -24 * (A.double().abs() @ B.double().abs().T) + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23) * exact.abs()
    assert bool(((whole[:, col:col + N].double() - exact).abs() <= bound).all())
    assert torch.equal(whole[:, :col], held[:, :col]) and torch.equal(whole[:, col + N:], held[:, col + N:])


@pytest.mark.parametrize("N", [192, 200, 248, 40])
def test_block_scaled_rows_of_any_alignment(N):
    g = torch.Generator(device=DEV).manual_seed(N)
    a, b = (torch.randn(n, 256, generator=g, device=DEV).bfloat16() for n in (200, N))
    aq, sa = mx.quantize_mx(a, sf_rows=256)
    bq, sb = mx.quantize_mx(b, sf_rows=mx._pad128(N + mx.TILE_N))
    got = mx.gemm_mx(aq, sa, bq, sb)
    L.check_status()
    da, db = mx.dequantize_mx(aq, mx.unpack_scales(sa, 200, 256)).double(), mx.dequantize_mx(bq, mx.unpack_scales(sb, N, 256)).double()
    exact = da @ db.T
    # (the tensor cores keep fewer bits of a sum than fp32 where operands are 8 bits wide: 2^-13 of the largest term is beyond what they drop)
    bound = 256 * 2.0 ** -22 * (da.abs() @ db.abs().T) + 2.0 ** -8 * exact.abs()
    assert bool(((got.double() - exact).abs() <= bound).all())


# groups of no rows (first, among others, last), of one reduction step and of several; outputs of one pair's tile and past it, on both sides of half a tile
@pytest.mark.parametrize("dtype,acc", [(torch.bfloat16, False), (torch.bfloat16, True), (torch.float32, False), (torch.float32, True)])
@pytest.mark.parametrize("M,N", [(64, 72), (128, 256), (136, 264), (384, 520)])
def test_grouped_reductions(M, N, dtype, acc):
    from dew_b200.ops import grouped
    rows = [0, 128, 64, 0, 0, 704, 128, 0]
    offsets = [sum(rows[:i]) for i in range(len(rows) + 1)]
    g = torch.Generator(device=DEV).manual_seed(M + N)
    dy, x = (torch.randn(offsets[-1] + 128, n, generator=g, device=DEV).bfloat16() for n in (M, N))      # rows behind the last group belong to none
    out = torch.randn(len(rows), M, N, generator=g, device=DEV).to(dtype)
    held = out.double()

    class Layout:
        pass
    layout = Layout()
    layout.offsets = torch.tensor(offsets, dtype=torch.int32, device=DEV)
    grouped.tgmm(dy, x, layout, len(rows), out=out, accumulate=acc)
    L.check_status()
    for i, (a, b) in enumerate(zip(offsets, offsets[1:])):
        exact = dy[a:b].double().T @ x[a:b].double() + (held[i] if acc else 0)
        size = dy[a:b].double().abs().T @ x[a:b].double().abs()
        # fp32 sums of (b - a) exact products in some order, and one rounding of the result
        bound = (b - a) * 2.0 ** -24 * size + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23) * exact.abs()
        assert bool(((out[i].double() - exact).abs() <= bound).all()), i


# less than a wave of tiles: reductions on both sides of the line where pairs take them, outputs within one tile's rows, past them, and not of whole pieces
@pytest.mark.parametrize("M,N,K", [(2048, 2048, 2040), (2048, 2048, 2048), (1096, 2312, 2056), (200, 16392, 4096), (128, 16384, 2304), (130, 9992, 2304)])
def test_pairs_below_a_wave(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(K)
    A, B = (torch.randn(n, K, generator=g, device=DEV).bfloat16() for n in (M, N))
    got = ops.gemm(A, B, out_dtype=torch.float32)
    L.check_status()
    assert torch.equal(got, ops.gemm(A, B, out_dtype=torch.float32, kernel="sm100_tcgen05", max_ctas=148))       # either kernel's sums are in the same order


# the same groups and parts by either kind of CTAs: outputs within one tile's rows and past them, rows and columns to spare
@pytest.mark.parametrize("paired", [False, True])
@pytest.mark.parametrize("dtype,acc", [(torch.bfloat16, False), (torch.bfloat16, True), (torch.float32, False), (torch.float32, True)])
@pytest.mark.parametrize("M,N", [(72, 264), (384, 520)])
def test_reductions_by_either_kind(M, N, dtype, acc, paired, monkeypatch):
    from dew_b200.ops import functional, grouped
    monkeypatch.setattr(grouped, "pairs_reduce", lambda *a: paired)
    test_grouped_reductions(M, N, dtype, acc)
    g = torch.Generator(device=DEV).manual_seed(M)
    for K, parts in ((2056, 2), (4096, 3)):
        monkeypatch.setattr(functional, "split_reduction", lambda *a: (parts, paired))
        A, B = torch.randn(K, M, generator=g, device=DEV).bfloat16(), torch.randn(N, K, generator=g, device=DEV).bfloat16()
        held = torch.randn(M, N, generator=g, device=DEV).to(dtype)
        out = held.clone()
        ops.gemm(A, B, a_mn=True, out=out, accumulate=acc, kernel="sm100_tcgen05")
        L.check_status()
        exact = A.double().T @ B.double().T + (held.double() if acc else 0)
        # fp32 sums of K exact products in some order, and one rounding of the result
        bound = K * 2.0 ** -24 * (A.double().abs().T @ B.double().abs().T) + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23) * exact.abs()
        assert bool(((out.double() - exact).abs() <= bound).all())
