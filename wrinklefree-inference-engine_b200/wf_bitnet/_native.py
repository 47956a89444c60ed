"""libwf_torch.so: the tensor-level calls as native torch ops (csrc/torch_ops.cpp).  Loading it registers the CUDA kernels of
torch.ops.sgl_kernel.bitnet_{gemv,gemm,quantize_activations}* and the torch.ops.wf_native ops."""
from __future__ import annotations

import torch

from . import _lib

TORCH_LIB_PATH = _lib.LIB_PATH.parent / "libwf_torch.so"
_ops = None


def _fake_linear(x, w, tile, N, K, w_scale):
    return x.new_empty(x.shape[0], N, dtype=torch.float32)


def _fake_mlp(x, gate_up_tile, N2, down_w, gate_scale, up_scale, down_scale, norm, eps):
    return x.new_empty(x.shape[0], down_w.shape[0], dtype=torch.bfloat16)


def _fake_attn(q, pool, max_pages, layers, kv_heads, page_size, head_dim, kv_dtype, layer, block_table, seq_lens, scale, out_dtype):
    return q.new_empty(q.shape, dtype=out_dtype)


def ops():
    """torch.ops.wf_native; raises when the library has not been built."""
    global _ops
    if _ops is None:
        if not TORCH_LIB_PATH.exists():
            raise _lib.WfError(f"{TORCH_LIB_PATH} not found: build it with `make -C {_lib.LIB_PATH.parent / 'csrc'}` (or __graft_entry__.build()). "
                               "There is no CPU fallback.")
        torch.ops.load_library(str(TORCH_LIB_PATH))
        for name, fake in (("linear", _fake_linear), ("mlp", _fake_mlp), ("paged_decode_attn", _fake_attn)):
            torch.library.register_fake(f"wf_native::{name}", fake)
        _ops = torch.ops.wf_native
    return _ops
