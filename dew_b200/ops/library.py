"""ctypes binding to ``libdewb.so`` (the sm_100a kernels) and the device status word.

The library is built in-tree by :mod:`dew_b200.ops.build`.  On a machine with a GPU every op in
:mod:`dew_b200.ops` runs through it; if it is missing there the ops raise instead of silently falling back,
so a GPU test can never pass on an eager path by accident.  On a CPU-only machine the ops use their
PyTorch reference implementations and this module is never loaded.
"""
from __future__ import annotations

import ctypes
import os
import threading
from pathlib import Path
from typing import Dict, Optional

import torch

_LIB: Optional[ctypes.CDLL] = None
_LIB_PATH = Path(__file__).resolve().parent / "libdewb.so"
_STATUS: Dict[int, torch.Tensor] = {}

ERROR_NAMES = {0: "ok", 1: "wait for a TMA stage timed out", 2: "wait for a free stage timed out",
               3: "wait for an accumulator timed out", 4: "wait for a drained accumulator timed out",
               5: "wait for a peer's flag timed out", 6: "bad argument", 7: "wait timed out"}


class KernelError(RuntimeError):
    """A launcher refused its arguments or a kernel reported a timed-out wait."""


class LibraryMissing(RuntimeError):
    pass


def path() -> Path:
    return _LIB_PATH


def exists() -> bool:
    return _LIB_PATH.exists()


def load(build_if_missing: bool = False) -> ctypes.CDLL:
    global _LIB
    if _LIB is not None:
        return _LIB
    if not _LIB_PATH.exists():
        if build_if_missing:
            from . import build
            build.build(verbose=False)
        else:
            raise LibraryMissing(f"{_LIB_PATH} is not built; run `python -m dew_b200.ops.build`")
    _LIB = _declare(ctypes.CDLL(str(_LIB_PATH)))
    return _LIB


# Argument types of the launchers that small steps call most: p a pointer, l a 64-bit and i a 32-bit integer, f a float.  A declared launcher takes Python numbers
# as they are; the others are given ctypes objects by their callers.
_SIGNATURES = {
    "dewb_rmsnorm_fwd": "pppppp" + "lifi" + "p",
    "dewb_ada_fwd": "ppppp" + "l" + "ppp" + "lii" + "f" + "p",
    "dewb_gemm_rows_bf16": "pppp" + "iii" + "lll" + "p",
    "dewb_swiglu_fwd": "ppp" + "lil" + "p",
    "dewb_time_features": "pp" + "iii" + "ff" + "p",
    "dewb_rope": "pppp" + "liiiif" + "p",
    "dewb_rope_rows": "ppp" + "liiiiif" + "p",
    "dewb_rmsnorm_bwd": "pppppppppppi" + "li" + "p",
    "dewb_swiglu_bwd": "ppppp" + "lil" + "p",
    "dewb_ce_rows": "pppp" + "lil" + "ifffi" + "p",
    "dewb_flash_fwd_var": "ppppp" + "iiiiii" + "l" * 12 + "f" + "iiiif" + "ppppp" + "pp",
    "dewb_flash_bwd_var": "pppppppppp" + "iiiiii" + "p" + "f" + "ii" + "f" + "pppp",
    "dewb_gemm_bf16": "ppp" + "iii" + "lll" + "iii" + "f" + "pip",
    "dewb_gemm_pair_bf16": "ppp" + "iii" + "lll" + "iii" + "f" + "pip",
    "dewb_gemm_bf16_bias": "pppp" + "iii" + "lll" + "iii" + "f" + "pip",
    "dewb_gemm_pair_bf16_bias": "pppp" + "iii" + "lll" + "iii" + "f" + "pip",
    "dewb_gemm_bf16_split": "pppp" + "iiiii" + "lll" + "iii" + "f" + "pp",
    "dewb_gemm_bf16_split_single": "pppp" + "iiiii" + "lll" + "iii" + "f" + "pp",
    "dewb_colsum_slabs": "li",
    "dewb_colsum_bf16": "ppp" + "lil" + "p",
    "dewb_ada_slab": "ii",
    "dewb_ada_bwd": "pppppp" + "l" + "ppppp" + "iiii" + "p",
    "dewb_rope_append": "pppp" + "iiiii" + "ppp" + "ii" + "p",
    "dewb_paged_decode_persist": "ppp" + "l" + "pppppppp" + "iiiiiii" + "f" + "iii" + "f" + "pp" + "l" + "i" + "pp",
}
_TYPES = {"p": ctypes.c_void_p, "l": ctypes.c_longlong, "i": ctypes.c_int, "f": ctypes.c_float}


def _declare(lib: ctypes.CDLL) -> ctypes.CDLL:
    for name, kinds in _SIGNATURES.items():
        if hasattr(lib, name):
            getattr(lib, name).argtypes = [_TYPES[k] for k in kinds]
    return lib


_ENV = getattr(os.environ, "_data", None)          # the environment as the bytes it is kept in
_ENCODED: Dict[str, object] = {}


def env(name: str, default: Optional[str] = None) -> Optional[str]:
    """``os.environ.get`` for names that every call looks up: ``os.environ`` encodes the name and raises an exception inside for each one that is not set, which
    takes longer than a launch."""
    if _ENV is None:
        return os.environ.get(name, default)
    key = _ENCODED.get(name)
    if key is None:
        key = _ENCODED[name] = os.environ.encodekey(name)
    value = _ENV.get(key)
    return default if value is None else os.environ.decodevalue(value)


def load_part(part: str) -> ctypes.CDLL:
    """Load the whole library if it is built, else the subset ``build.PARTS[part]``, building that where it is missing or out of date:
    for a program that runs from a source checkout and needs only those kernels."""
    global _LIB, _LIB_PATH
    if _LIB is None and not _LIB_PATH.exists():
        from . import build
        _LIB_PATH = build.build(verbose=False, part=part)
    return load()


def use_cuda(*tensors: torch.Tensor) -> bool:
    """True when the op must run on the CUDA library (all tensors on a GPU)."""
    for t in tensors:
        if isinstance(t, torch.Tensor):
            break
    else:
        return False
    if not t.is_cuda or env("DEWB_FORCE_REFERENCE") == "1":
        return False
    if _LIB is None:
        load()  # raises LibraryMissing on a machine with a GPU and no build
    ensure_device(t)
    return True


def unrecorded(*tensors: Optional[torch.Tensor]) -> bool:
    """Whether a call on these tensors leaves no trace in autograd, forward-mode differentiation, a functorch transform or a trace, so that its launches may run
    without an autograd node around them (the node alone takes as long as two launches)."""
    if torch.is_grad_enabled():
        for t in tensors:
            if t is not None and t.requires_grad:
                return False
    return plain_autograd()


def plain_autograd() -> bool:
    """Neither forward-mode differentiation, nor a functorch transform, nor a trace is under way."""
    return torch.autograd.forward_ad._current_level < 0 and not torch._C._are_functorch_transforms_active() and torch._C._get_tracing_state() is None


_TLS = threading.local()


def ensure_device(t: torch.Tensor) -> None:
    """Make ``t``'s device current for the library's own CUDA runtime on this thread (autograd runs backward on
    worker threads where nothing has selected a device yet)."""
    idx = t.get_device()
    if idx < 0:
        idx = torch.cuda.current_device()
    if getattr(_TLS, "device", None) != idx:
        check(load().dewb_set_device(ctypes.c_int(idx)), "set_device")
        _TLS.device = idx


def stream() -> int:
    """The current stream of the current device."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def stream_ptr() -> ctypes.c_void_p:
    return ctypes.c_void_p(stream())


def ptr(t: Optional[torch.Tensor]) -> ctypes.c_void_p:
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def at(t: Optional[torch.Tensor]) -> int:
    """A tensor's address for a declared launcher."""
    return 0 if t is None else t.data_ptr()


def status(device: Optional[torch.device] = None) -> torch.Tensor:
    """The per-device int32 status word kernels write a non-zero code into when a bounded wait gives up."""
    idx = torch.cuda.current_device() if device is None else (device.index or 0)
    if idx not in _STATUS:
        _STATUS[idx] = torch.zeros(1, dtype=torch.int32, device=f"cuda:{idx}")
    return _STATUS[idx]


def check_status(device: Optional[torch.device] = None) -> None:
    """Synchronising read of the status word; raises if any kernel reported an error since the last check."""
    word = status(device)
    code = int(word.item())
    if code != 0:
        word.zero_()
        raise KernelError(f"device kernel reported: {ERROR_NAMES.get(code, code)}")


NO_PAIRS = -6          # of the products' launchers: clusters of two CTAs cannot be placed on this device (lone CTAs then take the product)


def check(rc: int, what: str) -> None:
    if rc != 0:
        raise KernelError(f"{what}: launcher returned {rc}")


LAUNCHES = 0


def count_launches(n: int = 1) -> None:
    """Bookkeeping of how many of this library's kernels were launched (bench.py reports it)."""
    global LAUNCHES
    LAUNCHES += n
