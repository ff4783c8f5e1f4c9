"""Loader of the in-tree native library (``fluidmoe_b200/_C*.so``).

On a machine with a GPU the CUDA kernels are the only implementation of the hot ops, so a
missing library is an error there; on a CPU-only machine the pure-PyTorch reference path is
used instead and ``available()`` is False.
"""
from __future__ import annotations

import importlib
import os
import sysconfig

import torch

_C = None
_ERR = None
_STAMP = None      # of the library's file, when it was loaded or failed to load
_CUDA_SEEN = False
_FILE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "_C" + sysconfig.get_config_var("EXT_SUFFIX"))


def _file_stamp():
    try:
        st = os.stat(_FILE)
    except OSError:
        return None
    return st.st_ino, st.st_size, st.st_mtime_ns


def _try_load():
    """Load the library once.  A failure lasts as long as the file that caused it: a process may import the package,
    build the library and go on."""
    global _C, _ERR, _STAMP
    if _C is not None:
        return
    stamp = _file_stamp()
    if _ERR is not None and stamp == _STAMP:
        return
    _STAMP = stamp
    try:
        importlib.invalidate_caches()      # the folder may have been listed before the file was there
        _C = importlib.import_module("fluidmoe_b200._C")
        _ERR = None
    except Exception as e:  # noqa: BLE001 - recorded and re-raised by lib()
        _ERR = e


def is_current() -> bool:
    """Whether the loaded library is the one that is now in the package's folder."""
    return _C is not None and _STAMP == _file_stamp()


def available() -> bool:
    """True when the native library is importable *and* a CUDA device is present."""
    _try_load()
    return _C is not None and _cuda_present()


def _cuda_present() -> bool:
    # torch.cuda.is_available() asks the driver on every call; a device that was seen once stays
    global _CUDA_SEEN
    if not _CUDA_SEEN:
        _CUDA_SEEN = torch.cuda.is_available()
    return _CUDA_SEEN


def lib():
    """Return the extension module; raise loudly when it cannot be loaded."""
    _try_load()
    if _C is None:
        raise RuntimeError(
            "fluidmoe_b200 native library is not built (run `python -m fluidmoe_b200.build`): "
            f"{_ERR!r}"
        )
    return _C


def use_native(*tensors) -> bool:
    """Decide the code path for an op: CUDA tensors -> native kernels (mandatory), CPU -> torch."""
    if not tensors:
        return False
    for t in tensors:
        if t is not None and not t.is_cuda:
            return False
    lib()  # raises if missing: never fall back silently on a GPU box
    return True


def tensor_call(namespace: dict, name: str):
    """The native call ``name`` that takes tensors (csrc/tensor_calls.cpp), kept by a module as its global ``_<name>``.
    Such a call returns None for arguments it does not know, and the caller goes on with its own checks.  What a module
    keeps at first is a stand-in that finds the call when it is first used and takes its own place in ``namespace`` with
    it: importing the package loads no library, so that the library can be built by a process that has imported it."""
    key = "_" + name

    def first_use(*args):
        call = getattr(lib(), name, None)
        if call is None:
            raise RuntimeError("fluidmoe_b200 native library is older than the package (run `python -m fluidmoe_b200.build`)")
        if namespace.get(key) is first_use:
            namespace[key] = call
        return call(*args)
    return first_use


def stream_ptr() -> int:
    """Raw handle of the current stream of the current device (read afresh on every call; building the
    Python stream object for it took 5 us, a fifth of a short layer's host time)."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())
