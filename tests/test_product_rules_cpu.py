"""Which kernel a product of a size gets: the rules themselves, and where they lead, on the CPU."""
import pytest
import torch

from dew_b200.ops import functional as Fn
from dew_b200.ops import library as L

SMS = 148
up = lambda a, b: -(-a // b)
lone_tiles = lambda M, N: up(M, 128) * up(N, 256)
pair_tiles = lambda M, N: up(M, 256) * up(N, 256)


# odd numbers of row blocks and many columns: one wave of lone CTAs, two of pairs
@pytest.mark.parametrize("M,N,K", [(1152, 4096, 4096), (1025, 4096, 14336), (640, 7168, 4096), (384, 12288, 4096), (300, 12288, 4096), (384, 11264, 8192), (128, 19200, 4096), (128, 32768, 8192)])
def test_pairs_make_no_second_wave(M, N, K):
    assert lone_tiles(M, N) <= SMS < 2 * pair_tiles(M, N) and not Fn.pairs_below_a_wave(M, N, K)


class Launchers:
    """Stands in for the library: notes what is launched."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def launch(*args):
            self.calls.append(name)
            return 0
        return launch


@pytest.fixture
def launched(monkeypatch):
    def made():
        lib = Launchers()
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
    # a bias is added by the kernel that makes the whole product: no parts, so the line for pairs is that of unsplit ones
    (1024, 768, 3072, dict(bias=True), "dewb_gemm_bf16_bias"), (512, 3072, 12288, dict(bias=True), "dewb_gemm_pair_bf16_bias"), (1536, 1536, 16384, dict(bias=True), "dewb_gemm_pair_bf16_bias"),
    (1152, 4096, 4096, dict(bias=True), "dewb_gemm_bf16_bias"), (1536, 1536, 16384, dict(max_ctas=100), "dewb_gemm_bf16")])
def test_products_get_their_kernels(launched, M, N, K, kw, kernel):
    calls = launched()
    product(M, N, K, **kw)
    assert [c for c in calls if "gemm" in c] == [kernel]
