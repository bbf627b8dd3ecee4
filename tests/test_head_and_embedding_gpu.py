"""The gradients of the table at either end of a decoder: sums of looked-up rows, and the scaled weight gradient of the head."""
import pytest
import torch

from dew_b200 import ops
from dew_b200.ops import functional
from dew_b200.ops import library as L

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


def embedding_gradient(dy, ids, V):
    dw = torch.empty(V, dy.shape[1], dtype=torch.bfloat16, device=DEV)
    scratch = torch.empty(3 * ids.numel(), dtype=torch.int32, device=DEV)
    L.ensure_device(dy)
    L.check(L.load().dewb_embed_grad(L.ptr(dy), L.ptr(ids), L.ptr(dw), L.ptr(scratch), functional.c_int(ids.numel()), functional.c_int(dy.shape[1]), functional.c_ll(V),
                                     L.stream_ptr()), "embed_grad")
    return dw


# slices of the count of one token to sixteen; runs of one token, of a handful, of all; widths of one piece, past a block's columns, of both
@pytest.mark.parametrize("T,V,d", [(1, 1, 8), (3, 2, 1032), (255, 300, 64), (1024, 1, 128), (1025, 7, 8), (4096, 50000, 256), (16384, 256, 16), (0, 5, 8)])
def test_embedding_gradient(T, V, d):
    """The tokens' rows are summed in fp32 and rounded to bf16 once."""
    g = torch.Generator(device=DEV).manual_seed(T)
    ids, dy = torch.randint(0, V, (T,), generator=g, device=DEV), torch.randn(T, d, generator=g, device=DEV).bfloat16()
    got = embedding_gradient(dy, ids, V)
    want = torch.zeros(V, d, dtype=torch.float64, device=DEV).index_add_(0, ids, dy.double())
    size = torch.zeros(V, d, dtype=torch.float64, device=DEV).index_add_(0, ids, dy.double().abs())
    assert bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + T * 2.0 ** -24 * size).all())
    assert torch.equal(got, embedding_gradient(dy, ids, V))


# runs of as many tokens as one block takes, one more, up to and past the next multiples of it; at the front, behind others, at the end; columns short of and past a chunk
@pytest.mark.parametrize("d", [8, 72, 1032])
@pytest.mark.parametrize("runs", [[64], [65], [1, 64, 65, 1], [63, 66, 127, 2, 129], [30, 64, 64, 65, 300], [128, 128], [5] * 40 + [1000] + [3] * 20 + [70, 4096], [16384]])
def test_embedding_gradient_of_long_runs(runs, d):
    g = torch.Generator(device=DEV).manual_seed(len(runs) + d)
    ids = torch.repeat_interleave(torch.arange(len(runs), device=DEV) * 3, torch.tensor(runs, device=DEV))
    ids = ids[torch.randperm(len(ids), generator=g, device=DEV)].contiguous()
    dy = torch.randn(len(ids), d, generator=g, device=DEV).bfloat16()
    V = 3 * len(runs) + 1
    got = embedding_gradient(dy, ids, V)
    want, size = (torch.zeros(V, d, dtype=torch.float64, device=DEV).index_add_(0, ids, x) for x in (dy.double(), dy.double().abs()))
    assert bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + max(runs) * 2.0 ** -24 * size).all())
    assert torch.equal(got, embedding_gradient(dy, ids, V))


def test_padding_costs_no_more_than_tokens():
    """Half of a batch of one id: as many rows read and fewer written as where the ids differ, so at most as long but for the launches (twice, as a bound; a run that was
    summed by one block took nineteen times as long)."""
    T, d, V = 8192, 2048, 32768
    g = torch.Generator(device=DEV).manual_seed(0)
    dy, ids = torch.randn(T, d, generator=g, device=DEV).bfloat16(), torch.randint(0, V, (T,), generator=g, device=DEV)
    padded = ids.clone()
    padded[T // 2:] = 0
    took = {}
    for name, which in (("differ", ids), ("padded", padded)):
        times = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            torch.cuda._sleep(500000)                            # (the launches are enqueued by the time the first one starts)
            a.record()
            embedding_gradient(dy, which, V)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        took[name] = sorted(times)[3]
    assert took["padded"] < 2 * took["differ"], took


def test_embedding_lookup_keeps_its_gradients():
    """Through the lookup itself: by size to either backward, under second derivatives, and for tables that the kernels do not take."""
    g = torch.Generator(device=DEV).manual_seed(0)
    ids = torch.randint(0, 100, (4, 1024), generator=g, device=DEV)
    for width, dtype in ((512, torch.bfloat16), (64, torch.bfloat16), (513, torch.bfloat16), (512, torch.float32)):
        table = torch.randn(100, width, generator=g, device=DEV).to(dtype).requires_grad_()
        up = torch.randn(4, 1024, width, generator=g, device=DEV).to(dtype)
        out = ops.embedding(ids, table)
        assert torch.equal(out, table.detach()[ids])
        want = torch.zeros(100, width, dtype=torch.float64, device=DEV).index_add_(0, ids.reshape(-1), up.double().reshape(-1, width))
        got, = torch.autograd.grad(out, table, up)
        assert got.dtype == dtype and float((got.double() - want).norm() / want.norm()) < 2.0 ** -8
    table = torch.randn(100, 512, generator=g, device=DEV).bfloat16().requires_grad_()
    up = torch.randn(4, 1024, 512, generator=g, device=DEV).bfloat16().requires_grad_()
    first, = torch.autograd.grad(ops.embedding(ids, table), table, up, create_graph=True)
    second, = torch.autograd.grad(first.float().square().sum(), up)
    assert second.shape == up.shape and float(second.abs().sum()) > 0


@pytest.mark.parametrize("n", [1, 7, 8, 9, 8 * 256 + 5, 1 << 20])
def test_scaled_cast(n):
    """The bits of the product and the conversion one after the other."""
    g = torch.Generator(device=DEV).manual_seed(n)
    x, s = torch.randn(n, generator=g, device=DEV), torch.tensor(1.0 / 3.0, device=DEV)
    x[0] = float("inf")
    assert torch.equal(functional._scaled(x, s, torch.bfloat16), (x * s).to(torch.bfloat16))


@pytest.mark.parametrize("T,chunk", [(96, 96), (96, 40), (5, 2)])
def test_head_gradient_over_chunks(T, chunk):
    """The first chunk's product writes the weight gradient, the others add to it; against 64 bits, with the logits' gradient rounded to bf16 as the head keeps it."""
    g = torch.Generator(device=DEV).manual_seed(T + chunk)
    d, V = 64, 512
    h, w = torch.randn(T, d, generator=g, device=DEV).bfloat16().requires_grad_(), (torch.randn(V, d, generator=g, device=DEV) * 0.1).bfloat16().requires_grad_()
    targets = torch.randint(0, V, (T,), generator=g, device=DEV)
    loss, live = ops.linear_cross_entropy(h, w, targets, chunk=chunk)
    gh, gw = torch.autograd.grad(loss / live, (h, w))
    leaves = [x.detach().double().requires_grad_() for x in (h, w)]
    truth = torch.nn.functional.cross_entropy(leaves[0] @ leaves[1].t(), targets)
    for a, b in zip((gh, gw), torch.autograd.grad(truth, leaves)):
        assert float((a.double() - b).norm() / b.norm()) < 2.0 ** -6
