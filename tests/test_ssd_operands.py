"""What the state space kernels are given: operands that broadcast, and those that do not belong together."""
import pytest
import torch

from dew_b200.ops import library as L
from dew_b200.ops import scan
from dew_b200.ops import ssd as K

SIZES = dict(B=2, T=70, H=4, G=2)
# each operand as it may be handed over where it is the same along an axis
FORMS = [dict(dt=(2, 70, 1)), dict(A=(1,)), dict(A=()), dict(A=(1, 1, 4)), dict(D=(1,)), dict(initial=(1, 4, 64, 128)), dict(initial=(2, 1, 64, 1)), dict(dt=(2, 70, 1), A=(1,))]


def _operands(device="cpu", **shapes):
    B, T, H, G = SIZES.values()
    g = torch.Generator().manual_seed(5)
    r = lambda name, *full: torch.randn(shapes.get(name, full), generator=g)
    x, Bm, Cm = r("x", B, T, H, 64), 0.5 * r("B", B, T, G, 128), 0.5 * r("C", B, T, G, 128)
    dt, A = torch.nn.functional.softplus(r("dt", B, T, H) - 3), -r("A", H).abs() - 0.1
    D, initial = r("D", H), 0.2 * r("initial", B, H, 64, 128)
    half = lambda t: t.to(device).bfloat16()
    return [half(x), dt.to(device), A.to(device), half(Bm), half(Cm), D.to(device), initial.to(device)]


@pytest.mark.parametrize("form", FORMS)
def test_the_kernels_get_whole_operands(form):
    x, dt, A, Bm, Cm, D, initial = _operands(**form)
    if A.dim() > 1:
        A = A.reshape(-1)
    got = K._sized(x, dt, A, Bm, Cm, D, initial)
    for t, given, size in zip(got, (dt, A, D, initial), ((2, 70, 4), (4,), (4,), (2, 4, 64, 128))):
        assert t.shape == size and t.is_contiguous() and t.dtype == torch.float32 and torch.equal(t, given.expand(size))


@pytest.mark.parametrize("form", [dict(dt=(2, 69, 4)), dict(dt=(2, 70, 3)), dict(A=(3,)), dict(D=(5,)), dict(initial=(2, 4, 64, 64)), dict(B=(2, 70, 1, 128)), dict(C=(2, 69, 2, 128)),
                                  dict(B=(1, 70, 2, 128), C=(1, 70, 2, 128))])
def test_operands_of_other_sizes_are_refused_on_the_host(form):
    with pytest.raises((ValueError, RuntimeError)):
        K._sized(*_operands(**form))


@pytest.mark.gpu
@pytest.mark.parametrize("form", FORMS)
def test_broadcast_operands_and_their_gradients(form):
    norm = lambda t: float(t.double().norm())
    leaves = [t.requires_grad_() for t in _operands("cuda", **form)]
    B, T, H, G = SIZES.values()
    sizes = [(B, T, H, 64), (B, T, H), (H,), (B, T, G, 128), (B, T, G, 128), (H,), (B, H, 64, 128)]
    whole = [t.detach().double().expand(s if t.dim() <= len(s) else t.shape).contiguous().requires_grad_() for t, s in zip(leaves, sizes)]
    (y, S), (ty, tS) = scan.ssd(*leaves), scan.ssd_chunked(*whole)
    # as in the test of whole operands: bf16 outputs are rounded once
    assert norm(y - ty) < 4e-3 * norm(ty) and norm(S - tS) < 4e-3 * norm(tS)
    dy = torch.randn(y.shape, generator=torch.Generator().manual_seed(1)).to("cuda").bfloat16()
    got, want = torch.autograd.grad(y, leaves, dy), torch.autograd.grad(ty, whole, dy.double())
    L.check_status()
    # The kernels' errors are those of the gradients of whole operands (bf16: rounded once; fp32: sums of fp32 products, A's of differences of larger ones).  A smaller
    # operand's gradient is a sum of those, of either sign: their errors add up while they themselves may cancel, so the bound goes by the whole gradient.
    for n, a, b in zip(("x", "dt", "A", "B", "C", "D", "initial"), got, want):
        want_a = b if b.shape == a.shape else b.sum_to_size(a.shape)
        assert norm(a - want_a) < {"x": 2.5e-3, "B": 2.5e-3, "C": 2.5e-3, "A": 3e-5}.get(n, 3e-6) * norm(b), (n, norm(a - want_a), norm(b))
