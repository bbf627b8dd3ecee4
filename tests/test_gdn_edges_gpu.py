"""The gated delta rule's kernels where their splits end: one token, chunks of which the last is short or alone in its pair, key heads shared by value heads."""
import pytest
import torch

from dew_b200.ops import gdn, scan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,Hk,with_state", [(1, 1, 1, 1, True), (1, 63, 2, 2, False), (2, 64, 1, 1, True), (1, 65, 2, 1, True), (1, 128, 3, 3, False),
                                                 (2, 129, 2, 1, False), (1, 191, 1, 1, True), (1, 321, 4, 2, True)])
def test_forward_and_gradients(B, T, H, Hk, with_state):
    torch.manual_seed(T)
    unit = lambda *s: torch.nn.functional.normalize(torch.randn(*s, device="cuda"), dim=-1).to(torch.bfloat16)
    q, k, v = unit(B, T, Hk, 128), unit(B, T, Hk, 128), torch.randn(B, T, H, 128, device="cuda").to(torch.bfloat16)
    g, beta = -0.3 * torch.rand(B, T, H, device="cuda"), torch.rand(B, T, H, device="cuda")
    s0 = 0.1 * torch.randn(B, H, 128, 128, device="cuda") if with_state else None
    do, dS = torch.randn_like(v), 0.1 * torch.randn(B, H, 128, 128, device="cuda")
    ours = [t.clone().requires_grad_() for t in (q, k, v, g, beta)] + [s0.clone().requires_grad_() if with_state else None]
    o, S = gdn.gated_delta_rule(*ours[:5], initial_state=ours[5])
    torch.autograd.backward([o, S], [do, dS])
    ref = [t.double().requires_grad_() for t in (q, k, v, g, beta)] + [s0.double().requires_grad_() if with_state else None]
    rep = H // Hk
    ro, rS = scan.gated_delta_rule_chunked(ref[0].repeat_interleave(rep, 2), ref[1].repeat_interleave(rep, 2), *ref[2:5], initial_state=ref[5])
    torch.autograd.backward([ro, rS], [do.double(), dS.double()])
    # W, U, P, Vn, both states and the four matrices of the backward are rounded to bf16 (2^-9 a value, independent): up to eight such roundings meet in a gradient, and
    # the substitution lets each act on the rows behind it, for which a factor of two stands
    for name, a, b in [("o", o, ro), ("S", S, rS)] + [(n, x.grad, y.grad) for n, x, y in zip(("dq", "dk", "dv", "dg", "dbeta", "dS0"), ours, ref) if x is not None]:
        a, b = a.detach().double(), b.detach().double()
        assert torch.isfinite(a).all(), name
        assert float((a - b).norm()) <= 2 * 8 ** 0.5 * 2 ** -8 * float(b.norm()) + 1e-6 * b.numel() ** 0.5, name
