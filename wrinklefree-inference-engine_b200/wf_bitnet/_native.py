"""libwf_torch.so: the tensor-level calls as native torch ops (csrc/torch_ops.cpp).  Loading it registers the CUDA kernels of
torch.ops.sgl_kernel.bitnet_{gemv,gemm,quantize_activations}* and the torch.ops.wf_native ops.

It lies beside libwf_bitnet.so and is linked against the torch it was built with.  Where there is none (WF_BITNET_LIB names a library elsewhere) or it
does not load (another torch), the same calls go through ctypes: the same kernels, about 12 us more host time a call."""
from __future__ import annotations

import warnings

import torch

from . import _lib

TORCH_LIB_PATH = _lib.LIB_PATH.parent / "libwf_torch.so"
_ops = None


class _Ctypes:
    """The wf_native ops on the functions of wf_bitnet.ops."""

    @staticmethod
    def linear(x, w, tile, N, K, w_scale):
        from . import ops
        q, act_scale, rowsum = ops.quantize_activations(x, per_token=False)
        return ops.ternary_linear(w if tile else w.contiguous(), N, K, q, layout="tile" if tile else "i2s", mode="linear", rowsum=rowsum, act_scale=act_scale,
                                  w_scale=w_scale, out_dtype=torch.float32)

    @staticmethod
    def mlp(x, gate_up_tile, N2, down_w, gate_scale, up_scale, down_scale, norm, eps):
        from . import ops
        q, s, rs = ops.quantize_activations(x, per_token=True)
        ws = torch.tensor([gate_scale, up_scale], dtype=torch.float32, device=x.device)
        h = ops.ternary_linear(gate_up_tile, N2, x.shape[1], q, mode="linear", rowsum=rs, act_scale=s, w_scale=ws, relu2_mul=True, out_dtype=torch.bfloat16)
        q, s, rs, _ = ops.rmsnorm_quant(h, norm, eps)
        ws = torch.tensor([down_scale], dtype=torch.float32, device=x.device)
        return ops.ternary_linear(down_w.contiguous(), down_w.shape[0], down_w.shape[1] * 4, q, layout="i2s", mode="linear", rowsum=rs, act_scale=s, w_scale=ws,
                                  out_dtype=torch.bfloat16)

    @staticmethod
    def paged_decode_attn(q, pool, max_pages, layers, kv_heads, page_size, head_dim, kv_dtype, layer, block_table, seq_lens, scale, out_dtype):
        from . import ops
        return ops.paged_decode_attn_ctypes(q, _lib.KvLayout(pool.data_ptr(), max_pages, layers, kv_heads, page_size, head_dim, kv_dtype), layer, block_table, seq_lens, scale,
                                            out_dtype)


def _fake_linear(x, w, tile, N, K, w_scale):
    return x.new_empty(x.shape[0], N, dtype=torch.float32)


def _fake_mlp(x, gate_up_tile, N2, down_w, gate_scale, up_scale, down_scale, norm, eps):
    return x.new_empty(x.shape[0], down_w.shape[0], dtype=torch.bfloat16)


def _fake_attn(q, pool, max_pages, layers, kv_heads, page_size, head_dim, kv_dtype, layer, block_table, seq_lens, scale, out_dtype):
    return q.new_empty(q.shape, dtype=out_dtype)


def _load():
    if not TORCH_LIB_PATH.exists():
        _lib.lib()                       # raises where there is no library at all
        why = f"{TORCH_LIB_PATH} not found (`make -C {_lib._PKG_ROOT / 'csrc'}` builds it)"
    else:
        try:
            torch.ops.load_library(str(TORCH_LIB_PATH))
        except OSError as e:
            why = f"{TORCH_LIB_PATH} does not load: {e}"
        else:
            for name, fake in (("linear", _fake_linear), ("mlp", _fake_mlp), ("paged_decode_attn", _fake_attn)):
                torch.library.register_fake(f"wf_native::{name}", fake)
            return torch.ops.wf_native
    warnings.warn(f"{why}; the BitNet ops call their kernels through ctypes")
    return _Ctypes


def ops():
    """torch.ops.wf_native, or the same functions through ctypes; raises when libwf_bitnet.so has not been built."""
    global _ops
    if _ops is None:
        _ops = _load()
    return _ops


def is_native() -> bool:
    return ops() is not _Ctypes
