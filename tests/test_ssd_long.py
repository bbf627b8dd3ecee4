"""The state space scan over more chunks than a grid's second dimension holds."""
import pytest
import torch

from dew_b200.ops import library as L
from dew_b200.ops import scan


@pytest.mark.gpu
def test_more_than_65535_chunks():
    T, cut = 65536 * 64 + 10, 65535 * 64
    g = torch.Generator(device="cuda").manual_seed(0)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    # one token's x, B and C for all of them (the kernels read them by strides), steps of their own
    x, Bm, Cm = (t.bfloat16().expand(1, T, -1, -1) for t in (r(1, 1, 2, 64), r(1, 1, 1, 128), r(1, 1, 1, 128)))
    dt, A = torch.nn.functional.softplus(r(1, T, 2) - 3), torch.tensor([-0.5, -8.0], device="cuda")
    with torch.no_grad():
        y, last = scan.ssd(x, dt, A, Bm, Cm)
        head, state = scan.ssd(x[:, :cut], dt[:, :cut], A, Bm[:, :cut], Cm[:, :cut])
        tail, end = scan.ssd(x[:, cut:], dt[:, cut:], A, Bm[:, cut:], Cm[:, cut:], initial_state=state)
    L.check_status()
    # the walk carries its fp32 state over a chunk's end as it hands it out: the same bits
    assert torch.equal(y[:, cut:], tail) and torch.equal(last, end) and torch.equal(y[:, cut - 64:cut], head[:, cut - 64:])
