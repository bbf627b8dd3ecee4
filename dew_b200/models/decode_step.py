"""A plain decoder's layers for one token of one to four rows, issued by one call (``csrc/kernels/decode_step.cu``).

The layers' own modules would launch the same kernels on the same operands; what the call leaves out is their way through the interpreter, which takes four times as long as
the kernels of a small decoder.  So it takes a step only where a module does nothing but that: layers of the common form, weights in one piece, nobody watching, and every
product one that the few-row kernel would get.  Everything is looked at, and every pointer taken, for each step anew.
"""
from __future__ import annotations

import ctypes
import math
from typing import Optional, Tuple

import torch

from ..nn.attention import SelfAttention
from ..nn.kv_cache import KVStore
from ..nn.layers import Linear, RMSNorm
from ..nn.mlp import SwiGLU
from ..ops import functional as ops
from ..ops import library as L
from ..utils.hooks import nobody_watches_all, runs_alone_by_itself

_p, _i, _f = ctypes.c_void_p, ctypes.c_int, ctypes.c_float


class _Layer(ctypes.Structure):
    _fields_ = [(n, _p) for n in ("in_norm", "qkv", "out", "post_norm", "gate_up", "down", "keys", "values", "sinks")] + \
               [("in_eps", _f), ("post_eps", _f)] + [(n, _i) for n in ("window", "max_parts", "ff")]


class _Call(ctypes.Structure):
    _fields_ = [(n, _p) for n in ("embedded", "stream0", "stream1", "branch", "normed", "packed", "attended", "gates", "active", "rstd", "cosb", "sinb", "positions", "lengths",
                                  "page_table", "part_m", "part_l", "part_acc", "arrivals", "err")] + \
               [("pool_tokens", ctypes.c_longlong), ("scale", _f)] + \
               [(n, _i) for n in ("rows", "width", "heads", "kv_heads", "dim", "table_rows", "page_size", "max_pages", "min_tiles", "ctas")]


MOST_ROWS = 4


def _weight(linear, device) -> Optional[torch.Tensor]:
    """The weight of a plain layer without a bias, if it is one piece of bf16."""
    if type(linear) is not Linear or linear.bias is not None or not runs_alone_by_itself(linear):
        return None
    w = linear._parameters["weight"]
    return w if w.dtype == torch.bfloat16 and w.device == device and w.is_contiguous() and w.data_ptr() % 16 == 0 else None


def _norm(norm, device) -> Optional[torch.Tensor]:
    if type(norm) is not RMSNorm or norm.around or norm.one or not runs_alone_by_itself(norm):
        return None
    w = norm._parameters["weight"]
    return w if w.dtype == torch.bfloat16 and w.device == device and w.is_contiguous() and w.data_ptr() % 16 == 0 else None


def _common_layer(layer) -> bool:
    return (layer.kind in ("attention", "local") and layer.tp is None and layer.cross is None and layer.streams is None and layer.layer_scale is None and not layer.sparse
            and not layer.parallel and layer.mixer_out_norm is None and layer.mlp_out_norm is None and layer.residual_multiplier == 1.0 and runs_alone_by_itself(layer))


def _common_mixer(m, store) -> bool:
    return (type(m) is SelfAttention and m.num_kv_heads == store.kv_heads and m.head_dim == store.head_dim == m.value_dim and m.causal and not m.softcap and m.q_norm is None
            and m.q_gain is None and m.temperature is None and m.chunk is None and not m.head_gate and m.own_kv and m.rotation is None and not m.keep_first and not m.unit_qk
            and m.conv is None and m.weighting == "softmax" and m.head_temperature is None and m.heads_bias is None and m.gate_proj is None and m.head_transform is None
            and m.rotary is True and m.own_rope is None and runs_alone_by_itself(m))


def takes(h: torch.Tensor, cos, positions, store) -> bool:
    """What can be said without a look at the layers."""
    return (type(store) is KVStore and h.dim() == 3 and 1 <= h.shape[0] <= MOST_ROWS and h.shape[1] == 1 and h.shape[0] == store.rows and h.dtype == torch.bfloat16
            and h.is_contiguous() and h.shape[2] % 8 == 0 and h.shape[2] <= 8192 and h.data_ptr() % 16 == 0 and L.use_cuda(h) and store.slots is None and store.kind == 0
            and store.dtype == torch.bfloat16 and store.row_ids is None and store.head_dim == 128 and store.page_size % 64 == 0 and store.device == h.device and cos is not None
            and positions is not None and positions.numel() == h.shape[0] and L.env("DEWB_DECODE", "stream") == "stream" and L.env("DEWB_DECODE_PERSIST", "1") == "1"
            and not torch.is_grad_enabled() and L.plain_autograd() and ops.few_row_products_declared() and nobody_watches_all() and hasattr(L.load(), "dewb_decode_step"))


def run(model, h: torch.Tensor, cos, sin, positions, store) -> Optional[Tuple[torch.Tensor, torch.Tensor]]:
    """``h [R, 1, d]`` through ``model.layers`` -> (stream, pending branch), or None where the layers go one by one."""
    from .causal_transformer import DecoderLayer
    if not takes(h, cos, positions, store):
        return None
    R, d, dev, n = h.shape[0], h.shape[2], h.device, len(model.layers)
    G, D = store.kv_heads, store.head_dim
    layers, held, H, most, parts, shapes = (_Layer * n)(), [], None, 0, 0, set()
    min_tiles = int(L.env("DEWB_DECODE_MIN_TILES", store.MIN_TILES))
    for i, (layer, at) in enumerate(zip(model.layers, layers)):
        if type(layer) is not DecoderLayer or not _common_layer(layer) or layer.index != i:
            return None
        mods = layer._modules
        mixer, mlp = mods.get("mixer"), mods.get("mlp")
        if not _common_mixer(mixer, store) or type(mlp) is not SwiGLU or mlp.activation != "silu" or not runs_alone_by_itself(mlp):
            return None
        H = mixer.num_heads if H is None else H
        ws = (_norm(mods.get("input_norm"), dev), _weight(mixer._modules.get("qkv_proj"), dev), _weight(mixer._modules.get("o_proj"), dev), _norm(mods.get("post_norm"), dev),
              _weight(mlp._modules.get("gate_up_proj"), dev), _weight(mlp._modules.get("down_proj"), dev))
        if mixer.num_heads != H or any(w is None for w in ws):
            return None
        n1, qkv, out, n2, gu, down = ws
        ff = down.shape[1]
        if (n1.shape != (d,) or n2.shape != (d,) or qkv.shape != ((H + 2 * G) * D, d) or out.shape != (d, H * D) or gu.shape != (2 * ff, d) or down.shape != (d, ff) or ff % 8):
            return None
        shapes.update((qkv.shape, out.shape, gu.shape, down.shape))
        window = mixer.window or 0
        at.max_parts = (-(-(min(store.max_len, window) if window else store.max_len) // 64)) // min_tiles + 2      # (one tile on top: a window may straddle a boundary)
        at.in_norm, at.qkv, at.out, at.post_norm, at.gate_up, at.down = (w.data_ptr() for w in ws)
        at.keys, at.values = store.k[i].data_ptr(), store.v[i].data_ptr()
        at.in_eps, at.post_eps, at.window, at.ff = mods["input_norm"].eps, mods["post_norm"].eps, window, ff
        sinks = mixer._parameters.get("sinks")
        if sinks is not None:
            held.append(sinks.detach().float().contiguous())                       # referenced until the launches are enqueued
            at.sinks = held[-1].data_ptr()
        most, parts = max(most, ff), max(parts, at.max_parts)
    if H % G or H // G > 8 or not all(ops._few_rows(R, N, K) for N, K in shapes):
        return None
    pos32, lens32 = store._step_ints(positions.reshape(-1))
    pm, pl, pa = store._partials(R * H * parts, D, dev)
    stream = torch.empty(2, R, 1, d, dtype=h.dtype, device=dev)
    branch = torch.empty_like(h)
    sizes = [R * d, R * (H + 2 * G) * D, R * H * D, R * 2 * most, R * most]
    offsets = [sum(-(-s // 64) * 64 for s in sizes[:k]) for k in range(len(sizes) + 1)]
    scratch = torch.empty(offsets[-1] + 2 * 64, dtype=h.dtype, device=dev)         # (the rows' 1 / rms last, fp32)
    base = scratch.data_ptr()
    normed, packed, attended, gates, active, rstd = (base + 2 * o for o in offsets)
    status = L.status(dev)
    call = _Call(embedded=h.data_ptr(), stream0=stream.data_ptr(), stream1=stream.data_ptr() + 2 * R * d, branch=branch.data_ptr(), normed=normed, packed=packed, attended=attended,
                 gates=gates, active=active, rstd=rstd, cosb=cos.data_ptr(), sinb=sin.data_ptr(), positions=pos32.data_ptr(), lengths=lens32.data_ptr(),
                 page_table=store.page_table.data_ptr(), part_m=pm.data_ptr(), part_l=pl.data_ptr(), part_acc=pa.data_ptr(), arrivals=store._row_arrivals(R * G, dev).data_ptr(),
                 err=status.data_ptr(), pool_tokens=store.pages * store.page_size, scale=1.0 / math.sqrt(D), rows=R, width=d, heads=H, kv_heads=G, dim=D,
                 table_rows=cos.shape[0], page_size=store.page_size, max_pages=store.max_pages, min_tiles=min_tiles, ctas=store._decode_ctas(dev))
    L.check(L.load().dewb_decode_step(layers, _i(n), ctypes.byref(call), L.stream_ptr()), "decode_step")
    L.count_launches(9 * n)
    ops.count_few_row_products(4 * n)
    return stream[0], branch
