"""The Mamba-2 state space kernels, forward and every gradient, against the chunked form in 64 bits."""
import pytest
import torch

from dew_b200.ops import library as L
from dew_b200.ops import scan

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


def rel_err(a, b):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


def _inputs(B, T, H, G, seed, with_state):
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)
    x, Bm, Cm = r(B, T, H, 64).bfloat16(), (0.5 * r(B, T, G, 128)).bfloat16(), (0.5 * r(B, T, G, 128)).bfloat16()
    dt = torch.nn.functional.softplus(r(B, T, H) - 3)
    A = -torch.rand(H, generator=g, device=DEV) * 15 - 0.1
    return [x, dt, A, Bm, Cm, r(H), 0.2 * r(B, H, 64, 128) if with_state else None]


# chunk edges; one token; heads per group from two to many; few and many CTAs (every slicing of the walk and of a group's heads); a state in and a gradient of the last one
@pytest.mark.parametrize("B,T,H,G,with_state", [(1, 1, 2, 1, False), (1, 63, 2, 1, True), (2, 64, 4, 2, False), (1, 65, 8, 1, True), (3, 200, 32, 1, True),
                                                (2, 321, 96, 2, False), (2, 130, 128, 1, True), (1, 1024, 16, 4, True)])
def test_ssd_forward_and_gradients(B, T, H, G, with_state):
    ins = _inputs(B, T, H, G, T + H, with_state)
    leaves = [None if t is None else t.clone().requires_grad_() for t in ins]
    truth = [None if t is None else t.double().requires_grad_() for t in ins]
    y, S = scan.ssd(*leaves)
    ty, tS = scan.ssd_chunked(*truth)
    # bf16 outputs (2^-9 relative to each value, about 1.7e-3 in the norm) of products whose weights and states were rounded to bf16 once
    assert rel_err(y, ty) < 4e-3 and rel_err(S, tS) < 4e-3
    g = torch.Generator(device=DEV).manual_seed(7)
    dy = torch.randn(y.shape, generator=g, device=DEV).bfloat16()
    dS = 0.1 * torch.randn(S.shape, generator=g, device=DEV) if with_state else None
    grads = lambda y, S, ls, d: torch.autograd.grad((y, S) if dS is not None else (y,), [t for t in ls if t is not None], (dy.to(d), dS.to(S.dtype)) if dS is not None else (dy.to(d),))
    got, want = grads(y, S, leaves, y.dtype), grads(ty, tS, truth, torch.float64)
    L.check_status()
    names = [n for n, t in zip(("x", "dt", "A", "B", "C", "D", "initial"), ins) if t is not None]
    # bf16 gradients: one rounding of the result.  fp32 gradients: sums of fp32 products; those of the decays are differences of sums up to ten times as large,
    # and A's of 64 or more of them
    limit = {"x": 2.5e-3, "B": 2.5e-3, "C": 2.5e-3, "dt": 3e-6, "A": 3e-5, "D": 3e-6, "initial": 3e-6}
    for n, a, b in zip(names, got, want):
        assert rel_err(a, b) < limit[n], (n, rel_err(a, b))


# either side of the lines between a CTA's quarter, half and all of a state's columns: 74, 185 and 296 rows of one walk, the same of both
@pytest.mark.parametrize("B,H", [(1, 37), (1, 74), (1, 92), (1, 93), (1, 185), (1, 186), (2, 148), (3, 99)])
def test_ssd_walks_by_quarters_halves_and_whole_states(B, H):
    test_ssd_forward_and_gradients(B, 130, H, 1, True)


def test_ssd_takes_views_other_types_and_repeats():
    x, dt, A, Bm, Cm, D, s0 = _inputs(2, 100, 4, 1, 3, True)
    y, S = scan.ssd(x, dt, A, Bm, Cm, D, s0)
    # a slice of one projection, as the mixer hands it over; a slice off a 16-byte boundary is copied
    for pad in (8, 3):
        wide = torch.cat([x.flatten(2), Bm.flatten(2), Cm.flatten(2), x.new_zeros(2, 100, pad)], -1)[..., : 4 * 64 + 256]
        xs, bs, cs = (t.unflatten(-1, s) for t, s in zip(wide.split([256, 128, 128], -1), ((4, 64), (1, 128), (1, 128))))
        yv, Sv = scan.ssd(xs, dt, A, bs, cs, D, s0)
        assert torch.equal(y, yv) and torch.equal(S, Sv)
    # fp32 inputs are differentiated in fp32
    leaves = [t.float().requires_grad_() for t in (x, dt, A, Bm, Cm, D, s0)]
    yf, _ = scan.ssd(*leaves)
    truth = [t.detach().double().requires_grad_() for t in leaves]
    ty, _ = scan.ssd_chunked(*truth)
    dy = torch.randn_like(yf)
    for a, b in zip(torch.autograd.grad(yf, leaves, dy), torch.autograd.grad(ty, truth, dy.double())):
        assert rel_err(a, b) < 3e-5
    # the same bits twice
    leaves = [t.clone().requires_grad_() for t in (x, dt, A, Bm, Cm, D, s0)]
    one, two = (torch.autograd.grad(scan.ssd(*leaves)[0], leaves, dy.bfloat16()) for _ in range(2))
    assert all(torch.equal(a, b) for a, b in zip(one, two))
    L.check_status()
