"""The transposed block-scaled quantiser and the small kernels of the token exchange."""
import ctypes

import pytest
import torch

from dew_b200.ops import library as L
from dew_b200.ops import mx

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


@pytest.mark.parametrize("G,N,K", [(1, 128, 64), (3, 256, 192), (2, 384, 1408), (5, 128, 136)])      # (the last one's width is not whole tiles: the copying route)
def test_transposed_quantiser_gives_the_bytes_of_quantising_the_transpose(G, N, K):
    g = torch.Generator(device=DEV).manual_seed(K)
    x = (torch.randn(G, N, K, generator=g, device=DEV) * torch.exp2(torch.randint(-30, 30, (G, N, 1), generator=g, device=DEV).float())).bfloat16()
    x[0, :32, 0] = 0                                   # a block of zeros, one with an infinity and one with a NaN
    x[0, 5, 1], x[0, 6, 2] = float("inf"), float("nan")
    rows = (G * K + 127) // 128 * 128 + 128
    q, sf = mx.quantize_mx_t(x, rows)
    want_q, want_sf = mx.quantize_mx(x.transpose(1, 2).contiguous().reshape(G * K, N), sf_rows=rows)
    assert torch.equal(q.view(torch.uint8), want_q.view(torch.uint8)) and torch.equal(sf, want_sf)


@pytest.mark.parametrize("pairs,k,d", [(1, 1, 8), (30, 3, 264), (96, 6, 2048)])
def test_pair_dots(pairs, k, d):
    g = torch.Generator(device=DEV).manual_seed(d)
    rows, dy = (torch.randn(n, d, generator=g, device=DEV).bfloat16() for n in (pairs, pairs // k))
    out = torch.empty(pairs, device=DEV)
    L.check(L.load().dewb_moe_pair_dots(L.ptr(rows), L.ptr(dy), L.ptr(out), ctypes.c_int(pairs), ctypes.c_int(k), ctypes.c_int(d), L.stream_ptr()), "moe_pair_dots")
    want = (rows.double() * dy.double().repeat_interleave(k, 0)).sum(-1)
    # fp32 sums of d exact products: a few roundings of numbers as large as sqrt(d)
    assert float((out - want).abs().max()) < 1e-5 * d ** 0.5


def test_zero_pads_touches_the_pads_alone():
    d, counts = 72, [0, 1, 127, 128, 130, 0, 5]
    offsets = [0]
    for c in counts:
        offsets.append(offsets[-1] + (c + 127) // 128 * 128)
    cap = offsets[-1] + 128
    rows = torch.ones(cap, d, device=DEV, dtype=torch.bfloat16)
    off, cnt = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in (offsets, counts))
    L.check(L.load().dewb_moe_zero_pads(L.ptr(rows), L.ptr(off), L.ptr(cnt), ctypes.c_int(len(counts)), ctypes.c_int(cap), ctypes.c_int(d), L.ptr(L.status(rows.device)),
                                        L.stream_ptr()), "moe_zero_pads")
    live = torch.ones(cap, dtype=torch.bool)
    for o, c, e in zip(offsets, counts, offsets[1:]):
        live[o + c:e] = False
    assert torch.equal((rows != 0).all(1).cpu(), live) and torch.equal((rows == 0).all(1).cpu(), ~live)


# reductions of one stage, of as many as the scales are fetched ahead, of one more, and past the ring; tiles with rows and columns to spare, more tiles than CTAs
@pytest.mark.parametrize("M,N,K", [(1, 192, 128), (130, 200, 512), (128, 384, 640), (300, 64, 768), (2048, 2112, 896)])
def test_block_scaled_product_by_stages(M, N, K):
    """Against the same numbers in 64 bits: fp32 sums rounded to bf16 once."""
    from dew_b200.ops import mx
    g = torch.Generator(device="cuda").manual_seed(M + K)
    a, b = (torch.randn(n, K, generator=g, device="cuda").mul(torch.rand(n, 1, generator=g, device="cuda") * 4).bfloat16() for n in (M, N))
    aq, sa = mx.quantize_mx(a, sf_rows=-(-M // 128) * 128)
    bq, sb = mx.quantize_mx(b, sf_rows=N + mx.TILE_N)
    out = mx.gemm_mx(aq, sa, bq, sb)
    L.check_status()
    full = [mx.dequantize_mx(q, mx.unpack_scales(s, q.shape[0], K)).double() for q, s in ((aq, sa), (bq, sb))]
    want = full[0] @ full[1].t()
    assert float((out.double() - want).norm() / want.norm()) < 2.0 ** -8
