"""The host wrappers' common cases in native code (csrc/host.cpp).

`module()` is the extension, ready for use, or None where it or libb200ops.so has not been built,
or where it cannot be loaded (it is built against one torch, which may have been replaced since):
the wrappers of `ops.py` / `backward.py` then serve every call themselves, on the same kernels.
"""

from __future__ import annotations

import importlib.util
import os
import warnings

from . import _abi

PATH = os.path.join(_abi.CSRC_DIR, "_b200host.so")

_module = None
_unloadable = None  # (path, modification time) of a file that has been tried and could not be loaded


def module():
    global _module, _unloadable
    if _module is None and os.path.exists(PATH) and os.path.exists(_abi.LIB_PATH):
        file = (PATH, os.path.getmtime(PATH))
        if file == _unloadable:
            return None
        from . import ops

        try:
            spec = importlib.util.spec_from_file_location("_b200host", PATH)
            native = importlib.util.module_from_spec(spec)
            spec.loader.exec_module(native)
            native.setup(_abi.lib()._handle, ops, _abi.check, ops.F32_SPLIT_MIN_MACS, ops.SPLITK_MIN_K, ops.SPLITK_MAX_OUTPUTS)
        except Exception as e:
            _unloadable = file
            warnings.warn(f"{PATH} cannot be used ({e}); calls go through the Python wrappers. Rebuild it: python -m backendbench_b200.build")
            return None
        _module = native
    return _module
