"""Loader of the in-tree torch extension `hccl_b200/lib/hccl_b200_torch.so` (built by `hccl_b200.utils.build.build_torch_ext()`)."""
from __future__ import annotations

import importlib.util
import os
import threading
from pathlib import Path

from . import _lib

_EXT = None
_LOCK = threading.Lock()
EXT_PATH = Path(__file__).resolve().parent / "lib" / "hccl_b200_torch.so"


def ext():
    global _EXT
    with _LOCK:
        if _EXT is None:
            _lib.lib()   # libhccl_b200.so first (RTLD_GLOBAL), the extension links against it
            if not EXT_PATH.exists():
                raise RuntimeError(f"{EXT_PATH} is missing: build it with `python -m hccl_b200.utils.build`")
            spec = importlib.util.spec_from_file_location("hccl_b200_torch", str(EXT_PATH))
            mod = importlib.util.module_from_spec(spec)
            spec.loader.exec_module(mod)
            _EXT = mod
    return _EXT


_OPS = False


def ops():
    """The extension for the operator calls, or None where it was not built or another flavor of the native library was asked for
    (HCCL_B200_LIB): the extension links against the release library, and a communicator belongs to the library that made it."""
    global _OPS
    if _OPS is False:
        _OPS = None if os.environ.get("HCCL_B200_LIB") or not EXT_PATH.exists() else ext()
    return _OPS
