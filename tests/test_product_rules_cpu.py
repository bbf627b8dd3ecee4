"""Which kernel a product of a size gets: the rules themselves, and where they lead, on the CPU."""
import random

import pytest
import torch

from dew_b200.ops import functional as Fn
from dew_b200.ops import grouped
from dew_b200.ops import library as L

SMS = 148
up = lambda a, b: -(-a // b)
lone_tiles = lambda M, N: up(M, 128) * up(N, 256)
pair_tiles = lambda M, N: up(M, 256) * up(N, 256)


# odd numbers of row blocks and many columns: one wave of lone CTAs, two of pairs
@pytest.mark.parametrize("M,N,K", [(1152, 4096, 4096), (1025, 4096, 14336), (640, 7168, 4096), (384, 12288, 4096), (300, 12288, 4096), (384, 11264, 8192), (128, 19200, 4096), (128, 32768, 8192)])
def test_pairs_make_no_second_wave(M, N, K):
    assert lone_tiles(M, N) <= SMS < 2 * pair_tiles(M, N) and not Fn.pairs_below_a_wave(M, N, K)


def test_rules_over_the_sizes():
    rng = random.Random(0)
    for _ in range(4000):
        M, N, K = (int(2 ** rng.uniform(*r)) for r in ((0, 13), (3, 15), (6, 16)))
        if Fn.pairs_below_a_wave(M, N, K):
            assert pair_tiles(M, N) <= SMS // 2 and K >= 4096
        parts, paired = Fn.split_reduction(M, N, K)
        assert parts == Fn.reduction_splits(M, N, K) and 1 <= parts <= 8
        if parts == 1:
            assert not paired
            continue
        per = up(up(K, parts), 64) * 64
        assert 2 * lone_tiles(M, N) <= SMS and (parts - 1) * per < K <= parts * per and K >= 1024 * parts
        if paired:                                                        # no longer waves than lone CTAs would have, whatever these split
            assert K > 2048 * parts
            least = min(up(lone_tiles(M, N) * s, SMS) / s for s in range(1, 9) if s <= max(1, K // 1024))
            assert up(pair_tiles(M, N) * parts, SMS // 2) / parts <= least / 0.85


class Launchers:
    """Stands in for the library: notes what is launched, and says that pairs cannot be placed where ``pairs`` is false."""

    def __init__(self, pairs):
        self.pairs, self.calls = pairs, []

    def __getattr__(self, name):
        def launch(*args):
            self.calls.append(name)
            return 0 if self.pairs or name not in ("dewb_gemm_pair_bf16", "dewb_gemm_pair_bf16_bias", "dewb_gemm_bf16_split", "dewb_tgmm_bf16") else -6
        return launch


@pytest.fixture
def launched(monkeypatch):
    def made(pairs=True):
        lib = Launchers(pairs)
        monkeypatch.setattr(L, "load", lambda *a: lib)
        monkeypatch.setattr(L, "use_cuda", lambda *a: True)
        monkeypatch.setattr(L, "stream", lambda *a: 0)
        monkeypatch.setattr(L, "stream_ptr", lambda *a: 0)
        monkeypatch.setattr(L, "status", lambda *a: torch.zeros(1, dtype=torch.int32))
        return lib.calls
    return made


def product(M, N, K, **kw):
    a, b = torch.empty(M, K, dtype=torch.bfloat16), torch.empty(N, K, dtype=torch.bfloat16)
    Fn.gemm(a, b, bias=torch.empty(N, dtype=torch.bfloat16) if kw.pop("bias", False) else None, **kw)


@pytest.mark.parametrize("M,N,K,kw,kernel", [
    (2048, 2048, 64, {}, "dewb_gemm_bf16"), (2048, 2048, 8192, {}, "dewb_gemm_pair_bf16"), (1152, 4096, 4096, {}, "dewb_gemm_bf16"), (2048, 2560, 64, {}, "dewb_gemm_pair_bf16"),
    (1536, 1536, 16384, {}, "dewb_gemm_bf16_split"), (384, 6144, 4096, {}, "dewb_gemm_bf16_split_single"), (1024, 768, 2048, {}, "dewb_gemm_bf16_split_single"),
    # a bias is added by the kernel that makes the whole product: no parts, so the line for pairs is that of unsplit ones
    (1024, 768, 3072, dict(bias=True), "dewb_gemm_bf16_bias"), (512, 3072, 12288, dict(bias=True), "dewb_gemm_pair_bf16_bias"), (1536, 1536, 16384, dict(bias=True), "dewb_gemm_pair_bf16_bias"),
    (1152, 4096, 4096, dict(bias=True), "dewb_gemm_bf16_bias"), (1536, 1536, 16384, dict(max_ctas=100), "dewb_gemm_bf16")])
def test_products_get_their_kernels(launched, M, N, K, kw, kernel):
    calls = launched()
    product(M, N, K, **kw)
    assert [c for c in calls if "gemm" in c] == [kernel]


@pytest.mark.parametrize("M,N,K,kw,kernel", [(2048, 2560, 64, {}, "dewb_gemm_bf16"), (2048, 2560, 64, dict(bias=True), "dewb_gemm_bf16_bias"), (1536, 1536, 16384, {}, "dewb_gemm_bf16_split_single")])
def test_lone_ctas_where_pairs_cannot_be_placed(launched, M, N, K, kw, kernel):
    calls = launched(pairs=False)
    product(M, N, K, **kw)
    assert [c for c in calls if "gemm" in c][-1] == kernel


def test_grouped_reductions_get_their_kernels(launched):
    layout = grouped.group_layout(torch.arange(8).repeat_interleave(512), 8)
    for pairs in (True, False):
        calls = launched(pairs)
        for M, N in ((256, 1024), (128, 256)):
            grouped.tgmm(torch.empty(layout.rows, M, dtype=torch.bfloat16), torch.empty(layout.rows, N, dtype=torch.bfloat16), layout, 8)
        assert calls == (["dewb_tgmm_bf16"] if pairs else ["dewb_tgmm_bf16", "dewb_tgmm_bf16_single"]) + ["dewb_tgmm_bf16_single"]
    assert not grouped.pairs_reduce(16 * 128, 512, 256, 16) and grouped.pairs_reduce(64 * 128, 2816, 2048, 64) and not grouped.pairs_reduce(64 * 128, 128, 768, 64)
