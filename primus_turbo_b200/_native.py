"""Loads the native host path (``csrc/torch_ops.cpp``) and decides when a call may take it.

The extension does what the Python wrappers in ``pytorch/kernels`` and the autograd Functions in ``pytorch/ops`` do
-- check, allocate, launch, save for backward -- without the interpreter in between.  Those remain for what needs
Python: traced calls, dispatch modes, tensor subclasses other than a cached weight, and per-kernel timing or NVTX
ranges (a backward pass whose forward pass ran before the recording began is timed natively).  An entry of the extension returns ``None`` for arguments it does not handle, and the caller goes on in Python.
"""

from __future__ import annotations

import importlib.util
from importlib.machinery import ExtensionFileLoader
from pathlib import Path

import torch

from primus_turbo_b200 import _lib

_PATH = Path(__file__).resolve().parent / "_C" / "ptb_torch.so"


def _load():
    if not _PATH.exists():
        raise ImportError(f"{_PATH} is missing: build it with `python -m primus_turbo_b200.build`")
    loader = ExtensionFileLoader("ptb_torch", str(_PATH))
    module = importlib.util.module_from_spec(importlib.util.spec_from_file_location("ptb_torch", _PATH, loader=loader))
    loader.exec_module(module)
    module.setup(_lib.PtbError, _lib.timed_region)
    module.set_check_status(_lib._DEBUG_STATUS)
    return module


ext = _load()
_lib._set_native_recording = ext.set_recording
ext.set_recording(_lib._event_log is not None)
_PLAIN = (torch.Tensor, torch.nn.Parameter)


def usable(t) -> bool:
    """Whether a call on ``t`` may run natively: a plain CUDA tensor, nothing tracing or recording the call."""
    return (
        not torch.compiler.is_compiling()
        and type(t) in _PLAIN
        and t.is_cuda
        and _lib._event_log is None
        and not _lib._NVTX
        and torch._C._len_torch_dispatch_stack() == 0
    )


__all__ = ["ext", "usable"]
