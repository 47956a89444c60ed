"""The torch ops behind the linears and the decode attention: what they raise, what they return under autograd, and the same calls where only
libwf_bitnet.so is at hand."""
import os
import shutil
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest
import torch

PKG = Path(__file__).resolve().parents[1] / "wrinklefree-inference-engine_b200"


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


def alone(tmp_path, code):
    """Runs code in a process whose library lies in a folder without libwf_torch.so."""
    shutil.copy(PKG / "libwf_bitnet.so", tmp_path)
    env = dict(os.environ, WF_BITNET_LIB=str(tmp_path / "libwf_bitnet.so"), PYTHONPATH=f"{PKG}:{Path(__file__).parent}")
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return r


def test_without_the_torch_library_the_calls_go_through_ctypes(tmp_path):
    r = alone(tmp_path, "import torch, sgl_kernel\nfrom wf_bitnet import _native\nassert not _native.is_native()\n"
                        "for n in ('bitnet_gemv', 'bitnet_gemm_cpu', 'bitnet_quantize_activations', 'bitnet_mlp_forward'):\n"
                        "    assert 'CUDA: registered' in torch._C._dispatch_dump_table('sgl_kernel::' + n)\n")
    assert "ctypes" in r.stderr


def results():
    """One call of each op on fixed inputs -> arrays."""
    import sgl_kernel  # noqa: F401
    from wf_bitnet import ops
    from wrinklefree_inference.kernels.bitnet_patch import BitNetLinearNative
    g = torch.Generator().manual_seed(3)
    packed = torch.randint(0, 256, (96, 64), generator=g, dtype=torch.uint8) & 0xAA          # codes 0 and 2
    other = torch.randint(0, 256, (96, 64), generator=g, dtype=torch.uint8) & 0xAA
    down = torch.randint(0, 256, (40, 32), generator=g, dtype=torch.uint8) & 0xAA
    gate = torch.randint(0, 256, (128, 64), generator=g, dtype=torch.uint8) & 0xAA
    up = torch.randint(0, 256, (128, 64), generator=g, dtype=torch.uint8) & 0xAA
    x = torch.randn(33, 256, generator=g)
    out = []
    lin = BitNetLinearNative(256, 96, packed.cuda(), torch.tensor([0.03]))
    for m in (1, 8, 33):
        out.append(lin(x[:m].cuda().requires_grad_()))
        assert not out[-1].requires_grad
    q8, s = torch.ops.sgl_kernel.bitnet_quantize_activations(x.cuda())
    out += [q8, s, torch.ops.sgl_kernel.bitnet_gemv(other.cuda(), q8[0].contiguous(), 0.02), torch.ops.sgl_kernel.bitnet_gemm(other.cuda(), q8, 0.02)]
    out.append(torch.ops.sgl_kernel.bitnet_mlp_forward(x.cuda().bfloat16(), gate.cuda(), up.cuda(), down.cuda(), 0.02, 0.03, 0.04, torch.ones(256).cuda()[:200], 1e-5))
    kv = ops.PagedKV(8, 1, 2, 16, 128)
    kv.pool.copy_(torch.randn(kv.pool.shape, generator=g))
    q = torch.randn(2, 4, 128, generator=g).bfloat16().cuda().requires_grad_()
    out.append(ops.paged_decode_attn(q, kv, 0, torch.tensor([[3, 1], [0, 7]], dtype=torch.int32).cuda(), torch.tensor([20, 32], dtype=torch.int32).cuda()))
    assert not out[-1].requires_grad
    return [t.float().cpu().numpy() for t in out]


@pytest.mark.gpu
def test_native_calls_equal_those_through_ctypes(tmp_path):
    native()
    mine = results()
    alone(tmp_path, "import numpy as np, test_native_ops as t\nfrom wf_bitnet import _native\n"
                    f"r = t.results()\nassert not _native.is_native()\nnp.savez({str(tmp_path / 'r.npz')!r}, *r)\n")
    theirs = np.load(tmp_path / "r.npz")
    for i, a in enumerate(mine):
        assert np.array_equal(a, theirs[f"arr_{i}"]), i


@pytest.mark.gpu
def test_calls_on_two_streams_keep_to_their_own_workspaces():
    """Products whose K range is split meet in a workspace: calls side by side on two streams give the bits of calls one after another."""
    native()
    g = torch.Generator().manual_seed(5)
    w = (torch.randint(0, 256, (2560, 640), generator=g, dtype=torch.uint8) & 0xAA).cuda()
    xs = [torch.randint(-127, 128, (m, 2560), generator=g, dtype=torch.int8).cuda() for m in (1, 12)]
    want = [torch.ops.sgl_kernel.bitnet_gemm(w, x, 0.01) for x in xs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[], []]
    for _ in range(50):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(torch.ops.sgl_kernel.bitnet_gemm(w, xs[i], 0.01))
    torch.cuda.synchronize()
    for i in range(2):
        assert all(torch.equal(y, want[i]) for y in got[i])
