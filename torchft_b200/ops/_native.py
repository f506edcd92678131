"""Loader of the native autograd nodes (``csrc/host/autograd.cc``).

They stand in front of the Python nodes of ``functional.py`` and ``attention.py`` for the plain case of a call
and return ``None`` for any other, which the Python node then takes.  Like the kernel library the module has no
fallback: where it was not built, using it raises.
"""

from __future__ import annotations

import ctypes
import importlib
import threading

import torch

from torchft_b200.utils import build as _build

from . import _lib

_lock = threading.Lock()
_module = None

_ENTRIES = ("tft_gemm2_bf16", "tft_gemm2_workspace", "tft_rmsnorm_bwd_parts", "tft_rmsnorm_fwd", "tft_rmsnorm_bwd", "tft_swiglu_fwd", "tft_swiglu_bwd",
            "tft_xent", "tft_attn_fwd_pair", "tft_attn_bwd_tmem")


def _status_address(device_index: int) -> int:
    return _lib.status_word(torch.device("cuda", device_index)).data_ptr()


def _load():
    global _module
    with _lock:
        if _module is None:
            path = _build.autograd_module_path()
            if not path.exists():
                raise _lib.KernelError(f"{path} is missing: run `python -m torchft_b200.utils.build` (or __graft_entry__.build())")
            from . import functional

            handle = _lib.lib()
            entries = {name: ctypes.cast(getattr(handle, name), ctypes.c_void_p).value for name in _ENTRIES}
            loaded = importlib.import_module("torchft_b200._autograd")
            mark = getattr(loaded, "torch_mark", "built against an unknown torch;")
            if mark != _build._torch_mark(torch.__version__):
                raise _lib.KernelError(f"{path} was {mark[:-1]}, but torch {torch.__version__} runs: rebuild it with "
                                       "`python -m torchft_b200.utils.build`")
            loaded.setup(entries, _lib.KernelError, _status_address, functional._weight_gradient, functional._main_grad_target)
            _lib.add_launch_counter(loaded.launches)
            _module = loaded
    return _module


def module():
    return _module if _module is not None else _load()
