"""libwf_torch.so: the tensor-level calls as native torch ops (csrc/torch_ops.cpp).  Loading it registers the CUDA kernels of
torch.ops.sgl_kernel.bitnet_{gemv,gemm,quantize_activations}* and the torch.ops.wf_native ops."""
from __future__ import annotations

import torch

from . import _lib

TORCH_LIB_PATH = _lib.LIB_PATH.parent / "libwf_torch.so"
_ops = None


def ops():
    """torch.ops.wf_native; raises when the library has not been built."""
    global _ops
    if _ops is None:
        if not TORCH_LIB_PATH.exists():
            raise _lib.WfError(f"{TORCH_LIB_PATH} not found: build it with `make -C {_lib.LIB_PATH.parent / 'csrc'}` (or __graft_entry__.build()). "
                               "There is no CPU fallback.")
        torch.ops.load_library(str(TORCH_LIB_PATH))
        _ops = torch.ops.wf_native
    return _ops
