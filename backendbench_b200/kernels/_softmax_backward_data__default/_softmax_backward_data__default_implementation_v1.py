"""aten._softmax_backward_data.default on B200: backward of aten._softmax.default.

Loaded by a BackendBench DirectoryBackend (BackendBench/backends/directory.py:47-100):
the folder name is the overload with "." spelt "__", the exported callable is
`<folder>_kernel_impl`. The arithmetic runs in libb200ops.so through the C-ABI,
which a plain call reaches straight from native code, every other one (subclasses, modes,
gradients, other devices) by way of the `b200::softmax_backward` operator and its host wrapper.
"""

import os
import sys

try:
    from backendbench_b200 import custom_ops as _custom_ops
except ImportError:  # loaded by path from outside the repository root
    sys.path.insert(0, os.path.abspath(os.path.join(os.path.dirname(__file__), "..", "..", "..")))
    from backendbench_b200 import custom_ops as _custom_ops


_b200_softmax_backward = _custom_ops.entry("softmax_backward")  # torch.ops.b200.softmax_backward
_softmax_backward_data__default_kernel_impl = _b200_softmax_backward
