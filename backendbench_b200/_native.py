"""The host wrappers' common cases in native code (csrc/host.cpp).

`module()` is the extension, ready for use, or None where it or libb200ops.so has not been built:
the wrappers of `ops.py` / `backward.py` then serve every call themselves, on the same kernels.
"""

from __future__ import annotations

import importlib.util
import os

from . import _abi

PATH = os.path.join(_abi.CSRC_DIR, "_b200host.so")

_module = None


def module():
    global _module
    if _module is None and os.path.exists(PATH) and os.path.exists(_abi.LIB_PATH):
        from . import ops

        spec = importlib.util.spec_from_file_location("_b200host", PATH)
        native = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(native)
        native.setup(_abi.lib()._handle, ops, _abi.check, ops.F32_SPLIT_MIN_MACS, ops.SPLITK_MIN_K, ops.SPLITK_MAX_OUTPUTS)
        _module = native
    return _module
