"""The public ternary and attention ops in a caller's CUDA graph, where each of them hangs on the kernel before it by a programmatic edge: inputs that other
kernels of the same graph write (on the capturing stream, and on a second stream that joins it), replays with other inputs, results equal to eager calls."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def packed(n, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = torch.randint(0, 3, (n, k // 128, 4, 32), generator=g, device="cuda", dtype=torch.uint8)
    return (c[:, :, 0] << 6 | c[:, :, 1] << 4 | c[:, :, 2] << 2 | c[:, :, 3]).reshape(n, k // 4)


def replays(fill, calls, sources):
    """fill(sources) writes the ops' inputs with torch kernels; calls: the ops.  Captured: fill, then every call twice, then a fill on a second stream, its join and every
    call again.  Three replays with new sources."""
    def body(side):
        out = []
        fill()
        for f in calls:
            out += [f(), f()]
        main = torch.cuda.current_stream()
        side.wait_stream(main)
        with torch.cuda.stream(side):
            fill(2)
        main.wait_stream(side)
        for f in calls:
            out.append(f())
        return out
    s, side = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(s):
        for _ in range(2):
            body(side)                                     # workspaces of this stream
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        got = body(side)
    for seed in range(3):
        g = torch.Generator(device="cuda").manual_seed(seed)
        for t in sources:
            t.copy_(torch.randn(t.shape, generator=g, device="cuda"))
        graph.replay()
        torch.cuda.synchronize()
        have = [t.clone() for t in got]
        want = []
        fill()
        for f in calls:
            w = f()
            want += [w, w]
        fill(2)
        want += [f() for f in calls]
        torch.cuda.synchronize()
        for i, (a, b) in enumerate(zip(have, want)):
            assert torch.equal(a, b), (seed, i, (a.float() - b.float()).abs().max().item())
    del graph


# one and two tokens, a batch, split K, mma.sync tiles, one CTA a tile, pairs
@pytest.mark.parametrize("m,n,k", [(1, 2560, 2560), (2, 640, 1152), (6, 2560, 2560), (24, 4096, 4096), (64, 6912, 1024), (128, 14336, 4096), (300, 6912, 2560)])
def test_ternary_products(m, n, k):
    from sgl_kernel.quantization import bitnet_gemm, bitnet_gemv
    from wf_bitnet import ops
    w = packed(n, k, n + k)
    tile = ops.i2s_to_tile(w)
    src = torch.randn(m, k, device="cuda")
    q, rs, sc = torch.empty(m, k, device="cuda", dtype=torch.int8), torch.empty(m, device="cuda", dtype=torch.int32), torch.empty(m, device="cuda")
    one = torch.tensor([0.02], device="cuda")

    def fill(times=1):
        q.copy_((src * 30 * times).clamp(-127, 127))
        rs.copy_(q.sum(1, dtype=torch.int32))
        sc.copy_(src.abs().amax(1) * times)
    calls = [lambda: bitnet_gemm(w, q, 0.5), lambda: ops.ternary_linear(tile, n, k, q, mode="linear", rowsum=rs, act_scale=sc, w_scale=one, out_dtype=torch.bfloat16)]
    if m == 1:
        calls.append(lambda: bitnet_gemv(w, q[0], 0.5))
    replays(fill, calls, [src])


@pytest.mark.parametrize("m", [1, 5, 64, 4100])
def test_quantised_layers(m):
    import sgl_kernel  # noqa: F401
    from wf_bitnet import ops
    from wrinklefree_inference.kernels.bitnet_patch import BitNetLinearNative
    n, k, f = 640, 1280, 512
    layer = BitNetLinearNative(k, n, packed(n, k, 1), torch.tensor([0.03], device="cuda"))
    gate, up, down = packed(f, k, 2), packed(f, k, 3), packed(k, f, 4)
    norm = torch.ones(f, device="cuda", dtype=torch.bfloat16)
    src = torch.randn(m, k, device="cuda")
    x = torch.empty(m, k, device="cuda", dtype=torch.bfloat16)

    def fill(times=1):
        x.copy_(src * times)
    replays(fill, [lambda: layer(x), lambda: torch.ops.sgl_kernel.bitnet_mlp_forward_cpu(x, gate, up, down, 0.02, 0.03, 0.04, norm, 1e-5),
                   lambda: ops.quantize_activations(x, per_token=True)[0], lambda: ops.quantize_activations(x)[0], lambda: ops.rmsnorm_quant(x, torch.ones_like(x[0]), 1e-5)[0]], [src])


@pytest.mark.parametrize("cache", [torch.bfloat16, torch.int8])
@pytest.mark.parametrize("b,ctx", [(1, 700), (3, 90), (20, 300)])
def test_decode_attention(b, ctx, cache):
    from wf_bitnet import ops
    H, G, blocks = 20, 5, (ctx + 15) // 16
    kv = ops.PagedKV(b * blocks, 1, G, 16, 128, dtype=cache)
    k, v = (torch.randn(b * ctx, G * 128, device="cuda").to(torch.bfloat16) for _ in range(2))
    table = torch.randperm(b * blocks, device="cuda").to(torch.int32).view(b, blocks)
    pos = torch.arange(ctx, device="cuda").repeat(b)
    pages = table[torch.arange(b, device="cuda").repeat_interleave(ctx), pos // 16].contiguous()
    slots = (pos % 16).to(torch.int32)
    seq = torch.full((b,), ctx, dtype=torch.int32, device="cuda")
    src = torch.randn(b, H, 128, device="cuda")
    qx = torch.empty(b, H, 128, device="cuda", dtype=torch.bfloat16)

    def fill(times=1):
        qx.copy_(src * times)
        ops.kv_scatter(kv, k * times, v * times, pages, slots, 0)
    replays(fill, [lambda: ops.paged_decode_attn(qx, kv, 0, table, seq)], [src])


def test_the_product_without_allocations():
    """wf_bitnet_gemm_static, which is there for captures: cleared scratch, split K, several calls that share it."""
    from wf_bitnet._lib import lib
    L = lib()
    shapes = [(1, 2560, 2560), (8, 2560, 6912), (64, 3840, 2560)]
    ws = [packed(n, k, n) for _, n, k in shapes]
    src = torch.randn(64, 6912, device="cuda")
    q = torch.empty(64, 6912, device="cuda", dtype=torch.int8)
    ys = [torch.empty(m, n, device="cuda") for m, n, _ in shapes]

    def fill(times=1):
        q.copy_((src * 30 * times).clamp(-127, 127))

    def call(i):
        m, n, k = shapes[i]
        rc = L.wf_bitnet_gemm_static(ws[i].data_ptr(), q.data_ptr(), 0.5, m, n, k, ys[i].data_ptr(), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0, L.wf_last_error()
        return ys[i].clone()
    replays(fill, [lambda i=i: call(i) for i in range(3)], [src])
