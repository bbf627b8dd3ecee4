"""Modulated layer norms and gated residuals of diffusion transformers (``csrc/kernels/ada_norm.cu``), and the fixed position table of a patch grid.

``h = x + gate * branch`` and ``y = norm(h) * (1 + scale) + shift`` over tokens ``[B, n, d]`` with one shift, scale and gate ``[B, d]`` per image: one kernel each
way on a GPU in bf16, the plain expressions elsewhere.  Parity: ``modulate`` and the gated residuals of src/dew/nn/dit.py:572-727.
"""
from __future__ import annotations

import ctypes
import math
from typing import Optional, Tuple

import torch
import torch.nn.functional as F

from . import library as L

c_ll, c_int = ctypes.c_longlong, ctypes.c_int
MAX_WIDTH = 2048


def modulate(x, shift, scale):
    return x * (1 + scale.unsqueeze(1)) + shift.unsqueeze(1)


def _usable(x: torch.Tensor, branch: Optional[torch.Tensor], *mods: torch.Tensor) -> bool:
    """Rows of one width in whole 16-byte pieces, and per image one row of every modulation, all at one stride (slices of one projection)."""
    if not (x.dim() == 3 and x.dtype == torch.bfloat16 and L.use_cuda(x) and hasattr(L.load(), "dewb_ada_fwd")):
        return False
    B, n, d = x.shape
    if d % 8 or d > MAX_WIDTH or not 0 < B < 65536 or n == 0 or (branch is not None and (branch.shape != x.shape or branch.dtype != x.dtype or branch.device != x.device)):
        return False
    stride = mods[0].stride(0)
    return stride % 8 == 0 and all(m.shape == (B, d) and m.dtype == x.dtype and m.device == x.device and m.stride(1) == 1 and m.stride(0) == stride
                                   and m.data_ptr() % 16 == 0 for m in mods)


def _rows(t: torch.Tensor) -> torch.Tensor:
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _forward(x, branch, gate, shift, scale, eps):
    """-> y, h, stats (None where there is no norm; h is x where there is no branch)."""
    B, n, d = x.shape
    norm = shift is not None
    h = x if branch is None else torch.empty_like(x)
    y = torch.empty_like(x) if norm else None
    stats = torch.empty(B * n, 2, dtype=torch.float32, device=x.device) if norm else None
    at = L.at
    L.check(L.load().dewb_ada_fwd(at(x), at(branch), at(shift), at(scale), at(gate), (gate if shift is None else shift).stride(0), 0 if branch is None else at(h), at(y), at(stats),
                                  B * n, n, d, eps, L.stream()), "ada_fwd")
    L.count_launches()
    return y, h, stats


def _gradients(h, branch, gate, scale, eps, dy, dh):
    """What the backward kernel computes, as expressions that can be differentiated again: -> gradients of x, branch, gate, shift, scale."""
    wide = torch.promote_types(h.dtype, torch.float32)
    row = lambda t: t.to(wide).unsqueeze(1)
    g = torch.zeros((), dtype=wide, device=h.device) if dh is None else dh.to(wide)
    dbranch = dgate = dshift = dscale = None
    if scale is not None:
        u = h.to(wide) - h.to(wide).mean(-1, keepdim=True)
        rstd = torch.rsqrt(u.square().mean(-1, keepdim=True) + eps)
        u, v = u * rstd, dy.to(wide)
        a = v * (1 + row(scale))
        g = g + rstd * (a - a.mean(-1, keepdim=True) - u * (a * u).mean(-1, keepdim=True))
        dshift, dscale = v.sum(1), (v * u).sum(1)
    if branch is not None:
        dbranch, dgate = row(gate) * g, (branch.to(wide) * g).sum(1)
    return tuple(None if t is None else t.to(h.dtype) for t in (g, dbranch, dgate, dshift, dscale))


class _Ada(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, branch, gate, shift, scale, eps):
        ctx.set_materialize_grads(False)
        y, h, stats = _forward(x, branch, gate, shift, scale, eps)
        ctx.save_for_backward(h, branch, gate, scale, stats)
        ctx.eps = eps
        if branch is None:
            return y
        return h if shift is None else (y, h)

    @staticmethod
    def backward(ctx, *grads):
        h, branch, gate, scale, stats = ctx.saved_tensors
        norm = scale is not None
        dy, dh = (grads[0], None) if branch is None else (None, grads[0]) if not norm else grads
        if norm and dy is None:
            dy = torch.zeros_like(h)
        if torch.is_grad_enabled():                          # (create_graph: the kernel's results would have no history)
            return (*_gradients(h, branch, gate, scale, ctx.eps, dy, dh), None)
        dy, dh = (None if t is None else _rows(t.to(h.dtype)) for t in (dy, dh))
        B, n, d = h.shape
        lib = L.load()
        slab = lib.dewb_ada_slab(B, n)
        sets = 2 * norm + (branch is not None)
        L.ensure_device(h)
        part = torch.empty(B, -(-n // slab), sets, d, dtype=torch.float32, device=h.device)
        dmod = torch.empty(B, sets, d, dtype=h.dtype, device=h.device)
        dx = torch.empty_like(h) if norm else dh
        dbranch = None if branch is None else torch.empty_like(h)
        at = L.at
        L.check(lib.dewb_ada_bwd(at(dy), at(dh), at(h), at(branch), at(scale), at(gate), (gate if scale is None else scale).stride(0), at(stats), at(dx), at(dbranch), at(part),
                                 at(dmod), B, n, d, slab, L.stream()), "ada_bwd")
        L.count_launches(2)
        return dx, dbranch, None if branch is None else dmod[:, 2 * norm], dmod[:, 0] if norm else None, dmod[:, 1] if norm else None, None


def _run(x, branch, gate, shift, scale, eps):
    x, branch = _rows(x), None if branch is None else _rows(branch)
    if L.unrecorded(x, branch, gate, shift, scale):
        y, h, _ = _forward(x, branch, gate, shift, scale, eps)
        return y if branch is None else h if shift is None else (y, h)
    return _Ada.apply(x, branch, gate, shift, scale, eps)


def ada_norm(x: torch.Tensor, shift: torch.Tensor, scale: torch.Tensor, eps: float = 1e-6) -> torch.Tensor:
    """``norm(x) * (1 + scale) + shift`` with the layer norm without weights."""
    if _usable(x, None, shift, scale):
        return _run(x, None, None, shift, scale, eps)
    return modulate(F.layer_norm(x, (x.shape[-1],), None, None, eps), shift, scale)


def gated_ada_norm(x: torch.Tensor, branch: torch.Tensor, gate: torch.Tensor, shift: torch.Tensor, scale: torch.Tensor, eps: float = 1e-6) -> Tuple[torch.Tensor, torch.Tensor]:
    """``h = x + gate * branch``; -> (``norm(h) * (1 + scale) + shift``, ``h``)."""
    if _usable(x, branch, shift, scale, gate):
        return _run(x, branch, gate, shift, scale, eps)
    h = x + gate.unsqueeze(1) * branch
    return modulate(F.layer_norm(h, (h.shape[-1],), None, None, eps), shift, scale), h


def gated_add(x: torch.Tensor, branch: torch.Tensor, gate: torch.Tensor) -> torch.Tensor:
    """``x + gate * branch``."""
    if _usable(x, branch, gate):
        return _run(x, branch, gate, None, None, 0.0)
    return x + gate.unsqueeze(1) * branch


def time_features(t: torch.Tensor, dim: int, max_period: float, scale: float, dtype: torch.dtype) -> Optional[torch.Tensor]:
    """``nn.layers.sinusoidal`` by one kernel, where a row of fp32 times on a GPU leaves no trace in autograd; None elsewhere."""
    if not (t.is_cuda and t.dtype == torch.float32 and t.dim() == 1 and t.is_contiguous() and dim >= 2 and t.numel() * dim < 1 << 30 and dtype in (torch.float32, torch.bfloat16)
            and L.unrecorded(t) and L.use_cuda(t) and hasattr(L.load(), "dewb_time_features")):
        return None
    out = torch.empty(t.shape[0], dim, dtype=dtype, device=t.device)
    L.check(L.load().dewb_time_features(t.data_ptr(), out.data_ptr(), int(dtype == torch.bfloat16), t.shape[0], dim, -math.log(max_period), scale, L.stream()), "time_features")
    L.count_launches()
    return out


def sincos_grid(h: int, w: int, dim: int, device, dtype) -> torch.Tensor:
    """``[h * w, dim]``: the fixed 2-D sine-cosine signal of ``nn.dit.sincos_2d``, made by one kernel where a GPU wants it in bf16."""
    from ..nn.dit import sincos_2d
    device = torch.device(device)
    if device.type == "cuda" and dtype == torch.bfloat16 and dim % 4 == 0 and h > 0 and w > 0 and h * w * dim < 1 << 31 and L.env("DEWB_FORCE_REFERENCE") != "1" \
            and hasattr(L.load(), "dewb_sincos_grid"):
        out = torch.empty(h * w, dim, dtype=dtype, device=device)
        L.ensure_device(out)
        L.check(L.load().dewb_sincos_grid(L.ptr(out), c_int(h), c_int(w), c_int(dim), L.stream_ptr()), "sincos_grid")
        L.count_launches()
        return out
    return sincos_2d(h, w, dim, device).to(dtype)
