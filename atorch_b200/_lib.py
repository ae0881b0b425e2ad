"""Loader for ``libatb.so`` (the sm_100a kernels of atorch_b200).

The library is built in-tree by :mod:`atorch_b200.build`. On a machine with a GPU a missing
library is an error (ops must never fall back silently to eager PyTorch); on a CPU-only machine
``lib()`` returns ``None`` and the ops use their PyTorch reference implementations, which is what
the CPU test-suite exercises.
"""
from __future__ import annotations

import ctypes
import importlib.util
import os
from pathlib import Path
from typing import Optional

import torch

_LIB_PATH = Path(__file__).resolve().parent / "_C" / "libatb.so"
_lib = None
_tried = False


class KernelError(RuntimeError):
    """A launcher rejected its arguments or a kernel reported a non-zero status."""


# Argument types of the launchers on the per-operator path (p: pointer, i: int, l: long long, f: float), checked against
# csrc/ by a test. They are called through csrc/launcher.c with plain Python numbers; the others, and all of them where that
# module has not been built for this Python, through ctypes.
SIGNATURES = {
    "atb_gemm_bf16_2cta": "ppppiiillliiiifiiplpp",
    "atb_gemm_bf16_2cta_grouped": "ppppiiillliiiifiiplpiiiiipp",
    "atb_gemm_bf16": "ppppiiillliiiifiiplpp",
    "atb_gemm_bf16_2cta_swiglu": "ppppiiillllpp",
    "atb_gemm_bf16_2cta_rope": "pppiiilllpppiiipp",
    "atb_moe_sort_ids": "piipppp",
    "atb_moe_gather_rows": "pppiiip",
    "atb_gemm_bf16_2cta_kgroups": "pppiiillpiiipp",
    "atb_head_sum": "ppppliip",
    "atb_embedding_bwd": "ppppiiiiip",
    "atb_gemm_bf16_2cta_ragged": "pppiiilllipiippp",
    "atb_norm_fwd": "ppppppppiifiip",
    "atb_norm_bwd": "pppppppppiiiiip",
    "atb_colsum": "ppiiiip",
    "atb_rope": "pppppliiilliip",
    "atb_swiglu_fwd": "pplillp",
    "atb_swiglu_bwd": "ppplillp",
    "atb_flash_fwd_v2": "pppppppiiiiilllifppip",
    "atb_flash_fwd": "pppppppiiiiilllifpp",
    "atb_flash_bwd_split": "ppppppppppppiiiiillllllifppii",
    "atb_invert_perm": "ppip",
    "atb_moe_gather_sum": "pppipiiip",
    "atb_moe_ungather": "ppppippiiip",
    "atb_row_intervals": "pppiiiipipiippiip",
}
_CTYPE = {"p": ctypes.c_void_p, "i": ctypes.c_int, "l": ctypes.c_longlong, "f": ctypes.c_float}

_ctypes_launches = 0
_NOT_LAUNCHES = {"atb_norm_bwd_parts", "atb_sumsq_parts", "atb_set_comm_wait_ns", "atb_noalloc_max_n",
                 "atb_embedding_bwd_scratch"}


def __getattr__(name):
    if name == "launch_count":       # kernels of this library launched so far in this process
        return _ctypes_launches + (0 if _lib is None or _lib.launcher is None else _lib.launcher.count())
    raise AttributeError(f"module {__name__!r} has no attribute {name!r}")


class _CountingLib:
    """The library's functions by name, each launcher counting its calls (one per kernel launch)."""

    def __init__(self, cdll, launcher):
        self._cdll = cdll
        self.launcher = launcher

    def __getattr__(self, name):     # once per name: the function becomes an attribute
        raw = getattr(self._cdll, name)
        if name in SIGNATURES and self.launcher is not None:
            fn = self.launcher.Launcher(ctypes.cast(raw, ctypes.c_void_p).value, SIGNATURES[name])
        elif name in _NOT_LAUNCHES:
            fn = raw
        else:
            if name in SIGNATURES:
                raw.argtypes = [_CTYPE[c] for c in SIGNATURES[name]]

            def fn(*a, _raw=raw):
                global _ctypes_launches
                _ctypes_launches += 1
                return _raw(*a)
        self.__dict__[name] = fn
        return fn

    def has(self, name) -> bool:
        return name in self.__dict__ or hasattr(self._cdll, name)


def _load_launcher():
    """The extension module next to the library (csrc/launcher.c), or None where this Python has none and cannot build it."""
    from . import build as _build

    if not _build.LAUNCHER.exists() and not (os.environ.get("ATB_AUTO_BUILD", "1") == "1" and _build.build_launcher()):
        return None
    spec = importlib.util.spec_from_file_location("_launcher", _build.LAUNCHER)
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return module


def lib_path() -> Path:
    return _LIB_PATH


def lib():
    """The loaded library, or None on a CPU-only machine."""
    global _lib, _tried
    if _lib is not None:
        return _lib
    if not torch.cuda.is_available():
        return None
    if _tried:
        raise KernelError(f"{_LIB_PATH} could not be loaded")
    _tried = True
    if not _LIB_PATH.exists():
        if os.environ.get("ATB_AUTO_BUILD", "1") == "1":
            from . import build as _build

            _build.build()
        else:
            raise KernelError(f"{_LIB_PATH} is missing: run `python -m atorch_b200.build`")
    _lib = _CountingLib(ctypes.CDLL(str(_LIB_PATH)), _load_launcher())
    return _lib


def have_kernels() -> bool:
    return lib() is not None


def use_kernels(*tensors: torch.Tensor) -> bool:
    """True when the CUDA kernels must be used for these tensors (all on a CUDA device)."""
    if not tensors:
        return False
    for t in tensors:
        if t is not None and not t.is_cuda:
            return False
    return lib() is not None


def ptr(t: Optional[torch.Tensor]) -> ctypes.c_void_p:
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def addr(t: Optional[torch.Tensor]) -> int:
    """Address of a tensor's data (0: none) for a launcher with a declared signature."""
    return 0 if t is None else t.data_ptr()


def stream() -> int:
    """Handle of the current stream of the current device (what ``torch.cuda.current_stream().cuda_stream`` is)."""
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device())


def stream_ptr() -> ctypes.c_void_p:
    return ctypes.c_void_p(stream())


def check(rc: int, what: str) -> None:
    if rc != 0:
        raise KernelError(f"{what}: launcher returned {rc}")


_status: dict = {}


def status_word(device: torch.device) -> torch.Tensor:
    """Per-device int32 word that kernels with bounded waits write an error code to."""
    key = device.index if device.index is not None else torch.cuda.current_device()
    t = _status.get(key)
    if t is None:
        t = torch.zeros(1, dtype=torch.int32, device=device)
        _status[key] = t
    return t


_status_addr: dict = {}


def status_addr(t: torch.Tensor) -> int:
    """Address of the status word of the device that ``t`` is on."""
    i = t.get_device()
    a = _status_addr.get(i)
    if a is None:
        a = _status_addr[i] = status_word(t.device).data_ptr()
    return a


def check_status(device: torch.device) -> None:
    """Synchronising check of the status word; raises if a bounded wait ran out."""
    t = status_word(device)
    v = int(t.item())
    if v != 0:
        t.zero_()
        raise KernelError(f"kernel status {v} (1 = wait timeout, 3 = TMEM allocation, 4 = peer timeout)")


DT = {torch.bfloat16: 0, torch.float16: 1, torch.float32: 2}
