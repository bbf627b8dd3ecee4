"""Mamba-2 SSD on the sm_100a kernels (``csrc/kernels/ssd_sm100.cu``): state dimension 128, head dimension 64.

Forward: the states between the chunks of 64 tokens (sequential, one CTA per batch row, head and slice of columns), then the outputs of all chunks at once.
Backward, for bf16 inputs: the states again (nothing but the inputs is kept between the passes) and their gradients by the same walk in reverse, in fp32, then the
gradients of all chunks at once.  Inputs of other types are rounded to bf16 on the way forward and differentiated as they are: the loop-free chunked form in
PyTorch (``ops.scan.ssd_chunked``) is re-evaluated under autograd.  Reference: src/dew/nn/kernels/mamba_ssd.py (ChunkCumsum, BmmChunk, ChunkState, StatePassing,
ChunkScan), src/dew/nn/mixers/mamba2.py:101 ``chunk_ssd``.
"""
from __future__ import annotations

import ctypes

import torch

from . import library as L

CHUNK = 64
HEAD, STATE = 64, 128


def kernel_available(x: torch.Tensor, Bm: torch.Tensor) -> bool:
    H, P = x.shape[2], x.shape[3]
    G, N = Bm.shape[2], Bm.shape[3]
    return (x.is_cuda and P == HEAD and N == STATE and H % 2 == 0 and H % G == 0 and (H // G) % 2 == 0 and L.exists()
            and hasattr(L.load(), "dewb_ssd_fwd"))


def _rows(t: torch.Tensor) -> torch.Tensor:
    """``t [B, T, heads, width]`` in bf16 as the kernels take it: a token's heads in one piece, rows on 16-byte boundaries (a view of a wider projection is one)."""
    t = t.to(torch.bfloat16)
    inner = t.stride(3) == 1 and (t.shape[2] == 1 or t.stride(2) == t.shape[3])
    outer = all(n == 1 or s % 8 == 0 for n, s in zip(t.shape[:2], t.stride()))
    return t if inner and outer and t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.contiguous_format)


def _strides(*tensors: torch.Tensor):
    """Batch-row and token strides (0 where there is one)."""
    return (ctypes.c_longlong * (2 * len(tensors)))(*(s if n > 1 else 0 for t in tensors for n, s in zip(t.shape[:2], t.stride())))


def _sized(x, dt, A, Bm, Cm, D, initial):
    """dt ``[B, T, H]``, A and D ``[H]``, the initial state ``[B, H, 64, 128]``: in fp32, in these sizes, on ``x``'s device, as the kernels index them (what broadcasts
    to them is expanded; what does not is refused here, as are B and C of other sizes)."""
    B, T, H = x.shape[:3]
    if Bm.shape != Cm.shape or Bm.shape[:2] != x.shape[:2]:
        raise ValueError(f"ssd: x {tuple(x.shape)}, B {tuple(Bm.shape)} and C {tuple(Cm.shape)} do not belong together")
    for t in (dt, A, Bm, Cm, D, initial):
        if t is not None and t.dim() and t.device != x.device:
            raise ValueError(f"ssd: operands on {t.device} and on {x.device}")
    fp32 = lambda t, *size: None if t is None else t.detach().to(x.device).float().expand(size).contiguous()
    return fp32(dt, B, T, H), fp32(A, H), fp32(D, H), fp32(initial, B, H, HEAD, STATE)


def _forward(x, dt, A, Bm, Cm, D, initial):
    B, T, H, _ = x.shape
    dev = x.device
    chunks = -(-T // CHUNK)
    y = torch.empty(B, T, H, HEAD, dtype=torch.bfloat16, device=dev)
    last = torch.empty(B, H, HEAD, STATE, dtype=torch.float32, device=dev)
    states = torch.empty(B, H, chunks, HEAD, STATE, dtype=torch.bfloat16, device=dev)
    L.ensure_device(x)
    L.check(L.load().dewb_ssd_fwd(L.ptr(x), L.ptr(dt), L.ptr(A), L.ptr(Bm), L.ptr(Cm), L.ptr(D), L.ptr(initial), L.ptr(states), L.ptr(y), L.ptr(last),
                                  ctypes.c_int(B), ctypes.c_int(T), ctypes.c_int(H), ctypes.c_int(Bm.shape[2]), _strides(x, Bm, Cm), L.stream_ptr()), "ssd_fwd")
    L.count_launches(2)
    return y, last


def _backward(x, dt, A, Bm, Cm, D, initial, dy, dlast):
    """-> dx, ddt, dA, dB, dC, dD, dinitial."""
    B, T, H, _ = x.shape
    G, dev = Bm.shape[2], x.device
    chunks = -(-T // CHUNK)
    lib = L.load()
    f32 = dict(dtype=torch.float32, device=dev)
    splits = lib.dewb_ssd_splits(ctypes.c_int(B), ctypes.c_int(T), ctypes.c_int(H), ctypes.c_int(G))
    states, dstates = (torch.empty(B, H, chunks, HEAD, STATE, **f32) for _ in range(2))
    part = torch.empty(2, B * chunks, H, **f32)
    parts = torch.empty(2, splits, B, T, G, STATE, **f32) if splits > 1 else (None, None)
    dx = torch.empty(B, T, H, HEAD, dtype=torch.bfloat16, device=dev)
    dB, dC = (torch.empty(B, T, G, STATE, dtype=torch.bfloat16, device=dev) for _ in range(2))
    ddt, dA, dD = torch.empty(B, T, H, **f32), torch.empty(H, **f32), None if D is None else torch.empty(H, **f32)
    dinitial = torch.empty(B, H, HEAD, STATE, **f32)
    L.ensure_device(x)
    L.check(lib.dewb_ssd_bwd(L.ptr(x), L.ptr(dt), L.ptr(A), L.ptr(Bm), L.ptr(Cm), L.ptr(D), L.ptr(initial), L.ptr(dy), L.ptr(dlast), L.ptr(states), L.ptr(dstates),
                             L.ptr(part[0]), L.ptr(part[1]), L.ptr(parts[0]), L.ptr(parts[1]), L.ptr(dx), L.ptr(ddt), L.ptr(dA), L.ptr(dB), L.ptr(dC), L.ptr(dD),
                             L.ptr(dinitial), ctypes.c_int(B), ctypes.c_int(T), ctypes.c_int(H), ctypes.c_int(G), _strides(x, Bm, Cm), L.stream_ptr()), "ssd_bwd")
    L.count_launches(4)
    return dx, ddt, dA, dB, dC, dD, dinitial


class _SSD(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, dt, A, Bm, Cm, D, initial_state):
        ctx.set_materialize_grads(False)
        exact = all(t.dtype == torch.bfloat16 for t in (x, Bm, Cm))
        ctx.exact = exact
        dt32, A32, D32, initial32 = _sized(x, dt, A, Bm, Cm, D, initial_state)
        xb, bb, cb = _rows(x), _rows(Bm), _rows(Cm)
        ins = (dt32, A32, bb, cb, D32 if exact else None, initial32)
        y, last = _forward(xb, *ins)
        ctx.given = tuple(None if t is None else (t.dtype, t.shape) for t in (dt, A, D, initial_state))
        if exact:
            ctx.save_for_backward(xb, *ins)
        else:
            ctx.save_for_backward(x, dt, A, Bm, Cm, D, initial_state)
            if D is not None:
                y = (y.float() + x.float() * D.float()[None, None, :, None]).to(y.dtype)
        return y.to(x.dtype), last

    @staticmethod
    def backward(ctx, dy, dlast):
        saved = ctx.saved_tensors
        x = saved[0]
        dy = torch.zeros(x.shape, dtype=x.dtype, device=x.device) if dy is None else dy
        if not ctx.exact:
            from .scan import ssd_chunked
            with torch.enable_grad():
                leaves = [None if t is None else t.detach().requires_grad_(t.is_floating_point()) for t in saved]
                y, S = ssd_chunked(*leaves)
                need = [(t, i) for i, t in enumerate(leaves) if t is not None and ctx.needs_input_grad[i]]
                dlast = torch.zeros_like(S) if dlast is None else dlast
                grads = torch.autograd.grad((y, S), [t for t, _ in need], (dy.to(y.dtype), dlast.to(S.dtype)), allow_unused=True)
            out = [None] * 7
            for (t, i), g in zip(need, grads):
                out[i] = g
            return tuple(out)
        dy = dy.to(torch.bfloat16).contiguous()
        if dy.data_ptr() % 16:
            dy = dy.clone()
        dx, ddt, dA, dB, dC, dD, dinitial = _backward(*saved, dy, None if dlast is None else dlast.float().contiguous())
        fit = lambda g, given: None if given is None else g.sum_to_size(given[1]).to(given[0])
        dt_, A_, D_, initial_ = ctx.given
        return dx, fit(ddt, dt_), fit(dA, A_), dB, dC, fit(dD, D_), fit(dinitial, initial_)


def ssd(x, dt, A, Bm, Cm, D=None, initial_state=None):
    """x ``[B,T,H,64]``, dt ``[B,T,H]`` (after softplus), A ``[H]``, B / C ``[B,T,G,128]`` -> (y ``[B,T,H,64]``, state
    ``[B,H,64,128]`` fp32)."""
    if A.dim() > 1 and A.numel() == A.shape[-1]:
        A = A.reshape(-1)
    return _SSD.apply(x, dt, A, Bm, Cm, D, initial_state)
