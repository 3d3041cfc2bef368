"""ctypes loader for the in-tree CUDA kernel library (``dcp_b200/_kernels.so``).

The library exports a plain C ABI (``dcpk_*``); callers pass raw device pointers and the
current CUDA stream handle.  Loading fails loudly: on a machine with a GPU a missing library
is an error, never a silent fallback to eager PyTorch.
"""
from __future__ import annotations

import ctypes
import sysconfig
from pathlib import Path

import torch

_LIB = None


def lib_path() -> Path:
    return Path(__file__).resolve().parent.parent / "_kernels.so"


def load() -> ctypes.CDLL:
    global _LIB
    if _LIB is None:
        p = lib_path()
        if not p.exists():
            raise RuntimeError(
                f"{p} is missing: build it with `python -m dcp_b200.csrc.build` (needs nvcc, no GPU required)"
            )
        _LIB = ctypes.CDLL(str(p))
    return _LIB


def available() -> bool:
    return lib_path().exists()


def ptr(t) -> ctypes.c_void_p:
    """Device (or host) pointer of a torch tensor as a ctypes void pointer."""
    return ctypes.c_void_p(t.data_ptr())


def stream_handle():
    # the current stream of the current device; building a torch.cuda.Stream for it costs ten times as much, on
    # every launch
    return ctypes.c_void_p(torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice()))


LAUNCHES = 0  # kernel-entry calls made through this library since import (each launches >= 1 kernel)


def calls_path() -> Path:
    return lib_path().parent / ("_calls" + sysconfig.get_config_var("EXT_SUFFIX"))


def calls():
    """The native host side of single-rank attention calls (``csrc/host/calls.cpp``)."""
    load()
    try:
        from .. import _calls
    except ImportError as e:
        p = calls_path()
        if not p.exists():
            raise RuntimeError(f"{p} is missing: build it with `python -m dcp_b200.csrc.build`") from e
        # it is there: most likely built for another torch
        raise RuntimeError(f"{p} does not load with torch {torch.__version__} ({e}): rebuild it with "
                           "`python -m dcp_b200.csrc.build --force`") from e
    return _calls


def count(n: int):
    """``n`` kernel entries were called by native code."""
    global LAUNCHES
    LAUNCHES += n


def check(rc: int, what: str):
    global LAUNCHES
    LAUNCHES += 1
    if rc != 0:
        raise RuntimeError(f"{what} failed with code {rc}")
