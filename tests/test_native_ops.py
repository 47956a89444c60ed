"""The torch ops behind the linears and the decode attention: what they raise, what they return under autograd, and the same calls where only
libwf_bitnet.so is at hand."""

import pytest
import torch


def native():
    import sgl_kernel  # noqa: F401  the sgl_kernel schemas come first
    from wf_bitnet import _native
    assert _native.is_native()
    return _native.ops()


def test_missing_gpu_or_cpu_tensors_raise_as_through_ctypes():
    from wf_bitnet import _lib
    with pytest.raises(ValueError if _lib.available() else _lib.WfError):
        native().linear(torch.zeros(2, 128), torch.zeros(8, 32, dtype=torch.uint8), False, 8, 128, torch.ones(1))


def test_no_autograd_node_and_fakes():
    ops = native()
    for name in ("linear", "mlp", "paged_decode_attn"):
        assert "AutogradCUDA: fallthrough" in torch._C._dispatch_dump_table(f"wf_native::{name}")
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode():
        x = torch.empty(3, 128, device="cuda", dtype=torch.bfloat16)
        y = ops.linear(x, torch.empty(8, 32, device="cuda", dtype=torch.uint8), False, 8, 128, torch.empty(1, device="cuda"))
        assert y.shape == (3, 8) and y.dtype == torch.float32 and y.device.type == "cuda"
