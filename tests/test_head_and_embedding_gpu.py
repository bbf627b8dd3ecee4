"""The gradients of the table at either end of a decoder: sums of looked-up rows, and the scaled weight gradient of the head."""
import pytest
import torch

from dew_b200 import ops
from dew_b200.ops import functional
from dew_b200.ops import library as L

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


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
