"""Modulated norms and gated residuals, forward and every gradient, against the plain expressions in 64 bits."""
import math

import pytest
import torch
import torch.nn.functional as F

from dew_b200.nn.dit import ModulatedBlock, sincos_2d
from dew_b200.ops import ada
from dew_b200.ops import library as L

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


def rel_err(a, b):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


# one token, a warp's rows and one more, several slabs an image; every width a warp holds in 1, 2, 3, 4, 6 and 8 pieces a lane, full and partly filled
@pytest.mark.parametrize("B,n,d", [(1, 1, 8), (2, 9, 256), (3, 70, 264), (2, 64, 768), (1, 333, 1000), (2, 5, 1280), (1, 40, 2048)])
@pytest.mark.parametrize("form", ["norm", "both", "gate", "both, y unused", "both, h unused"])
def test_forward_and_gradients(B, n, d, form):
    g = torch.Generator(device=DEV).manual_seed(n + d)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV).bfloat16()
    x, branch, m = r(B, n, d) + 0.5, r(B, n, d), 0.5 * r(B, 3 * d)
    dy, dh = r(B, n, d), r(B, n, d)

    def run(x, branch, m, dt):
        shift, scale, gate = m.chunk(3, -1)
        if dt != torch.bfloat16:
            h = x if form == "norm" else x + gate.unsqueeze(1) * branch
            h = h + (h.detach().bfloat16().to(dt) - h.detach())                # (the stream carries h in bf16: what is normalised is what it carries)
            y = (h - h.mean(-1, keepdim=True)) * torch.rsqrt(h.var(-1, unbiased=False, keepdim=True) + 1e-6) * (1 + scale.unsqueeze(1)) + shift.unsqueeze(1)
            return (y,) if form == "norm" else (h,) if form == "gate" else (y, h)
        if form == "norm":
            return (ada.ada_norm(x, shift, scale),)
        return (ada.gated_add(x, branch, gate),) if form == "gate" else ada.gated_ada_norm(x, branch, gate, shift, scale)

    outs, grads = [], []
    for dt in (torch.bfloat16, torch.float64):
        leaves = [t.to(dt).requires_grad_() for t in (x, branch, m)]
        out = run(*leaves, dt)
        pairs = {"norm": [dy], "gate": [dh], "both": [dy, dh], "both, y unused": [None, dh], "both, h unused": [dy, None]}[form]
        kept = [(o, p.to(dt)) for o, p in zip(out, pairs) if p is not None]
        outs.append(out)
        grads.append(torch.autograd.grad([o for o, _ in kept], leaves, [p for _, p in kept], allow_unused=True))
    L.check_status()
    # one rounding of each result to bf16 (2^-9 of each value); h as it was rounded is the reference's as well, but beside a rounding boundary the fp32 sum may take the other side
    for a, b in zip(*outs):
        assert rel_err(a, b) < 4e-3
    for i, (a, b) in enumerate(zip(*grads)):
        assert (a is None) == (b is None) == (form == "norm" and i == 1)                  # (no branch in that form)
        if a is not None:
            assert rel_err(a, b) < 6e-3
    with torch.no_grad():
        assert all(torch.equal(a, b) for a, b in zip(run(x, branch, m, torch.bfloat16), outs[0]))


def test_position_table_and_a_hooked_norm():
    for h, w, d in ((3, 5, 4), (16, 16, 768), (7, 2, 36)):
        assert rel_err(ada.sincos_grid(h, w, d, DEV, torch.bfloat16), sincos_2d(h, w, d, DEV).bfloat16()) < 1e-4
    # a block whose norm is watched calls it
    block = ModulatedBlock(64, 1, dtype=torch.bfloat16, device=DEV)
    with torch.no_grad():
        for p in block.parameters():
            p.copy_(torch.randn_like(p) * 0.1)
        x, c = torch.randn(2, 128, 64, device=DEV).bfloat16(), torch.randn(2, 64, device=DEV).bfloat16()
        plain, seen = block(x, c), []
        handle = block.norm1.register_forward_hook(lambda *_: seen.append(1))
        hooked = block(x, c)
        handle.remove()
        assert seen == [1] and rel_err(hooked, plain) < 2e-2


@pytest.mark.parametrize("B,d,dtype", [(1, 2, torch.float32), (3, 7, torch.float32), (5, 256, torch.bfloat16), (64, 1153, torch.bfloat16), (0, 8, torch.bfloat16)])
def test_time_features(B, d, dtype):
    """Against 64 bits: an angle of up to 1000 turns on its fp32 roundings (the product with the frequency, and the frequency: some 2^-23 of it each), the rest on one
    rounding of the result; and a time that is differentiated keeps its graph."""
    from dew_b200.nn.layers import sinusoidal
    t = torch.rand(B, generator=torch.Generator(device=DEV).manual_seed(d), device=DEV) * 1000
    got = sinusoidal(t, d, scale=16.0 if d < 8 else 1.0, dtype=dtype)
    assert got.shape == (B, d) and got.dtype == dtype
    half = d // 2
    angle = t.double()[:, None] * (16.0 if d < 8 else 1.0) * torch.exp(-math.log(10000.0) * torch.arange(half, device=DEV, dtype=torch.float64) / half)
    want = torch.cat([angle.cos(), angle.sin(), angle.new_zeros(B, d % 2)], -1)
    bound = torch.cat([angle, angle, angle.new_zeros(B, d % 2)], -1) * 2.0 ** -20 + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -22)
    assert bool(((got.double() - want).abs() <= bound).all())
    leaf = t.clone().requires_grad_()
    assert B == 0 or float(torch.autograd.grad(sinusoidal(leaf, d, dtype=dtype).float().sum(), leaf)[0].abs().sum()) > 0


def test_blocks_share_the_activation_of_their_condition():
    """The same outputs whether the blocks make it themselves (somebody looks at them) or are given it."""
    from dew_b200.models import SimpleDiT
    torch.manual_seed(0)
    model = SimpleDiT(patch_size=2, emb_features=128, num_layers=3, num_heads=2, input_channels=4, output_channels=4, num_classes=10, dtype=torch.bfloat16, device=DEV)
    for p in model.parameters():
        torch.nn.init.normal_(p, std=0.05)
    x, t, label = torch.randn(2, 8, 8, 4, device=DEV), torch.rand(2, device=DEV), torch.tensor([1, 7], device=DEV)
    shared = model(x, t, {"label": label})
    hooks = [m.register_forward_hook(lambda *a: None) for m in (*model.blocks, model.output)]
    own = model(x, t, {"label": label})
    for h in hooks:
        h.remove()
    assert torch.equal(shared, own)
