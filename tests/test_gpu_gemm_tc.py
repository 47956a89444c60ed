"""GPU parity: the tcgen05 (kind::i8) prefill GEMM.  int32 accumulators bit-exact vs the oracle on sizes it
finishes in seconds, fused epilogues identical to the mma.sync path, and at the 2B prefill size
(8 x 2048 tokens) size-independent properties: equality with the already-pinned mma.sync kernel on the same
inputs, linearity in the activations and an oracle check of a random sample of rows."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def make(n, k, m, seed, raw=False):
    rng = np.random.default_rng(seed)
    w = rng.integers(-1, 2, size=(n, k)).astype(np.float32)
    packed = O.pack_ternary(w)[0]
    if raw:
        q = rng.integers(-128, 128, size=(m, k)).astype(np.int8)
        return packed, q, None, q.astype(np.int32).sum(1).astype(np.int32)
    x = (rng.standard_normal((m, k)) * 3).astype(np.float32)
    q, s, rs = O.quantize_act_i8_rows(x)
    return packed, q, s, rs


@pytest.mark.parametrize("nk", [(2560, 2560), (3840, 2560), (2560, 6912), (200, 640), (128, 128), (1000, 384)])
@pytest.mark.parametrize("m", [128, 130, 333, 512])
def test_tc_accumulators_bit_exact(nk, m):
    from wf_bitnet import ops
    n, k = nk
    packed, q, _, rs = make(n, k, m, n * 13 + k + m, raw=(m == 333))
    want = O.gemm_i32_fast(packed, q, 0)
    pi = cu(packed)
    tile = ops.i2s_to_tile(pi)
    for layout, wt in (("i2s", pi), ("tile", tile)):
        got = ops.ternary_linear(wt, n, k, cu(q), layout=layout, mode="i32_plus1", algo=3).cpu().numpy()
        assert np.array_equal(got, want), layout
    got = ops.ternary_linear(tile, n, k, cu(q), mode="i32", rowsum=cu(rs), algo=3).cpu().numpy()
    assert np.array_equal(got, O.gemm_i32_fast(packed, q, 1))


def test_tc_small_m_and_extremes():
    """M below one tile (TMA zero-fills the missing tokens) and the adversarial +-max inputs (|acc| = 2*128*K)."""
    from wf_bitnet import ops
    packed, q, _, _ = make(384, 512, 5, 3, raw=True)
    got = ops.ternary_linear(cu(packed), 384, 512, cu(q), layout="i2s", mode="i32_plus1", algo=3).cpu().numpy()
    assert np.array_equal(got, O.gemm_i32_fast(packed, q, 0))
    ones = cu(O.pack_ternary(np.ones((256, 28672), np.float32))[0])
    for val in (127, -128):
        a = torch.full((130, 28672), val, dtype=torch.int8, device="cuda")
        out = ops.ternary_linear(ones, 256, 28672, a, layout="i2s", mode="i32_plus1", algo=3)
        assert torch.all(out == 2 * val * 28672)


def test_tc_fused_epilogues_match_mma_path():
    from wf_bitnet import ops
    rng = np.random.default_rng(11)
    m, k, n, ffn = 300, 512, 640, 256
    packed, q, s, rs = make(n, k, m, 5)
    tile = ops.i2s_to_tile(cu(packed))
    ws = torch.tensor([0.7, 1.3, 2.1]).cuda()
    kw = dict(mode="linear", rowsum=cu(rs), act_scale=cu(s))
    a = ops.ternary_linear(tile, n, k, cu(q), w_scale=ws, seg_end=[384, 512, 640], out_dtype=torch.float32, algo=3, **kw)
    b = ops.ternary_linear(tile, n, k, cu(q), w_scale=ws, seg_end=[384, 512, 640], out_dtype=torch.float32, algo=2, **kw)
    assert torch.equal(a, b)
    from test_gpu_linear import ref_dequant          # the reference's fp32 rounding sequence (direct_inference_full.py:202-206)
    scale_n = np.concatenate([np.full(384, 0.7), np.full(128, 1.3), np.full(128, 2.1)]).astype(np.float32)
    assert np.array_equal(a.cpu().numpy(), ref_dequant(packed, q, rs, scale_n, s))
    res = torch.from_numpy(rng.standard_normal((m, n)).astype(np.float32) * 50).to(torch.bfloat16).cuda()
    w1 = torch.tensor([1.1]).cuda()
    a = ops.ternary_linear(tile, n, k, cu(q), w_scale=w1, residual=res, out_dtype=torch.bfloat16, algo=3, **kw)
    lin = torch.from_numpy(ref_dequant(packed, q, rs, np.float32(1.1), s)).to(torch.bfloat16)
    assert torch.equal(a.cpu(), res.cpu() + lin)
    wg = rng.integers(-1, 2, size=(ffn, k)).astype(np.float32)
    wu = rng.integers(-1, 2, size=(ffn, k)).astype(np.float32)
    pg, pu = O.pack_ternary(wg)[0], O.pack_ternary(wu)[0]
    tile_gu = ops.i2s_to_tile(ops.interleave_rows16(cu(pg), cu(pu)))
    sg, su = np.float32(0.9), np.float32(1.6)
    g = torch.from_numpy(ref_dequant(pg, q, rs, sg, s)).to(torch.bfloat16)
    u = torch.from_numpy(ref_dequant(pu, q, rs, su, s)).to(torch.bfloat16)
    got = ops.ternary_linear(tile_gu, 2 * ffn, k, cu(q), w_scale=torch.tensor([float(sg), float(su)]).cuda(), relu2_mul=True,
                             out_dtype=torch.bfloat16, algo=3, **kw).cpu()
    assert got.shape == (m, ffn) and torch.equal(got, torch.relu(g).square() * u)


@pytest.mark.parametrize("nk", [(3840, 2560), (2560, 6912)])
def test_tc_prefill_size_properties(nk):
    """A full prefill batch: M = 8 x 2048 tokens."""
    from wf_bitnet import ops
    n, k = nk
    m = 16384
    rng = np.random.default_rng(n)
    packed = O.pack_ternary(rng.integers(-1, 2, size=(n, k)).astype(np.float32))[0]
    tile = ops.i2s_to_tile(cu(packed))
    g = torch.Generator(device="cuda").manual_seed(1)
    q1 = torch.randint(-64, 64, (m, k), generator=g, device="cuda", dtype=torch.int8)
    q2 = torch.randint(-63, 64, (m, k), generator=g, device="cuda", dtype=torch.int8)
    y1 = ops.ternary_linear(tile, n, k, q1, mode="i32_plus1", algo=3)
    y2 = ops.ternary_linear(tile, n, k, q2, mode="i32_plus1", algo=3)
    y12 = ops.ternary_linear(tile, n, k, q1 + q2, mode="i32_plus1", algo=3)
    assert torch.equal(y1 + y2, y12)                                                   # linearity (exact integers)
    assert torch.equal(y1, ops.ternary_linear(tile, n, k, q1, mode="i32_plus1", algo=2))   # the pinned mma.sync kernel
    rows = rng.choice(m, size=64, replace=False)
    want = O.gemm_i32_fast(packed, q1[torch.from_numpy(rows).cuda()].cpu().numpy(), 0)
    assert np.array_equal(y1[torch.from_numpy(rows).cuda()].cpu().numpy(), want)       # oracle on a random sample of tokens


@pytest.mark.parametrize("m,n", [(130, 384), (500, 200), (64, 100), (129, 128)])
def test_tc_bf16_output_of_partial_tiles(m, n):
    """bf16 results with one weight scale where the last tile has fewer than 64 tokens or fewer than 32 rows: bit-equal to the rounding sequence."""
    from test_gpu_linear import ref_dequant
    from wf_bitnet import ops
    k = 512
    packed, q, s, rs = make(n, k, m, m + n)
    want = torch.from_numpy(ref_dequant(packed, q, rs, np.float32(1.7), s)).to(torch.bfloat16)
    got = ops.ternary_linear(ops.i2s_to_tile(cu(packed)), n, k, cu(q), mode="linear", rowsum=cu(rs), act_scale=cu(s), w_scale=torch.tensor([1.7]).cuda(),
                             out_dtype=torch.bfloat16, algo=3).cpu()
    assert torch.equal(got, want)


@pytest.mark.parametrize("m", [17, 33, 63, 65, 128, 129])
@pytest.mark.parametrize("nk", [(131, 1152), (2540, 2560), (96, 6912)])
def test_tc_shared_k_range(m, nk):
    """Few tokens: the K range of a tile shared by a cluster (unequal parts when K / 128 is no multiple of the cluster), every kind of output."""
    from test_gpu_linear import ref_dequant
    from wf_bitnet import ops
    n, k = nk
    packed, q, s, rs = make(n, k, m, n + k + m)
    pi, acc = cu(packed), O.gemm_i32_fast(packed, q, 0)
    want = acc.astype(np.float32) * np.float32(0.0123)
    assert np.array_equal(ops.bitnet_gemm(pi, cu(q), 0.0123).cpu().numpy(), want)
    kw = dict(layout="i2s", mode="linear", rowsum=cu(rs), act_scale=cu(s), algo=3)
    got = ops.ternary_linear(pi, n, k, cu(q), w_scale=torch.tensor([0.9]).cuda(), out_dtype=torch.bfloat16, **kw).cpu()
    assert torch.equal(got, torch.from_numpy(ref_dequant(packed, q, rs, np.float32(0.9), s)).to(torch.bfloat16))
    if n % 32 == 0:
        gu = ops.interleave_rows16(cu(packed[:n // 2]), cu(packed[n // 2:]))
        g = torch.from_numpy(ref_dequant(packed[:n // 2], q, rs, np.float32(0.9), s)).to(torch.bfloat16)
        u = torch.from_numpy(ref_dequant(packed[n // 2:], q, rs, np.float32(1.6), s)).to(torch.bfloat16)
        got = ops.ternary_linear(gu, n, k, cu(q), w_scale=torch.tensor([0.9, 1.6]).cuda(), relu2_mul=True, out_dtype=torch.bfloat16, **kw).cpu()
        assert torch.equal(got, torch.relu(g).square() * u)


# (N, K, tokens, tokens per tile of CTA pairs): every width; one k-block, a last weight load of one, two, three and four k-blocks; one round of tiles and several, at both depths of
# the operand ring (192 tokens and 256); rows and tokens that end inside a tile
PAIR_SHAPES = [(256, 128, 40, 32), (272, 640, 33, 32), (131, 384, 190, 32), (2560, 2560, 200, 32), (6912, 2560, 75, 64), (4090, 1152, 777, 96), (6912, 1152, 500, 128),
               (6905, 2560, 1987, 160), (13824, 2560, 300, 160), (8192, 896, 2500, 160), (6912, 128, 4000, 192), (6912, 640, 4000, 192), (2560, 6912, 1500, 256),
               (2560, 6912, 2700, 256)]


@pytest.mark.parametrize("nkm", PAIR_SHAPES)
def test_tc_pairs(nkm):
    """Every kind of output on CTA pairs, both weight layouts, bit-equal to the mma.sync kernel; accumulators of a sample of rows equal to the oracle's."""
    from wf_bitnet import ops
    from wf_bitnet._lib import lib
    n, k, m, tokens = nkm
    assert lib().wf_gemm_tc_pair_tokens(m, n, k, 3, 0) == tokens              # linear results
    rng = np.random.default_rng(n + k + m)
    q = torch.from_numpy(rng.integers(-128, 128, size=(m, k)).astype(np.int8)).cuda()
    code = rng.integers(0, 3, size=(n, k // 128, 4, 32)).astype(np.uint8)
    packed = (code[:, :, 0] << 6 | code[:, :, 1] << 4 | code[:, :, 2] << 2 | code[:, :, 3]).reshape(n, k // 4)
    pi = cu(packed)
    tile = ops.i2s_to_tile(pi)
    rs, sc = q.int().sum(1).int(), torch.rand(m, device="cuda") + 0.5
    rows = rng.choice(m, size=min(m, 24), replace=False)
    want = O.gemm_i32_fast(packed, q.cpu().numpy()[rows], 0)
    res = torch.randn(m, n, device="cuda").to(torch.bfloat16)
    one, two = torch.tensor([0.3], device="cuda"), torch.tensor([0.3, 0.2], device="cuda")
    lin = dict(mode="linear", rowsum=rs, act_scale=sc)
    forms = [dict(mode="i32", rowsum=rs), dict(lin, w_scale=one, out_dtype=torch.float32), dict(lin, w_scale=one, out_dtype=torch.bfloat16),
             dict(lin, w_scale=two, seg_end=[n // 2, n], out_dtype=torch.float32), dict(lin, w_scale=one, residual=res, out_dtype=torch.bfloat16)]
    if n % 32 == 0:
        forms += [dict(lin, w_scale=two, relu2_mul=True, out_dtype=torch.bfloat16), dict(lin, w_scale=two, relu2_mul=True, out_dtype=torch.float32)]
    for layout, wt in (("i2s", pi), ("tile", tile)):
        got = ops.ternary_linear(wt, n, k, q, layout=layout, mode="i32_plus1", algo=3).cpu().numpy()
        assert np.array_equal(got[rows], want), layout
        for f in forms:
            a, b = (ops.ternary_linear(wt, n, k, q, layout=layout, algo=x, **f) for x in (3, 2))
            assert torch.equal(a, b), (layout, list(f))
    assert torch.equal(ops.bitnet_gemm(pi, q, 0.0123).cpu()[rows], torch.from_numpy(want.astype(np.float32) * np.float32(0.0123)))


def test_a_wait_that_ran_out_is_reported_once():
    """The word that a product leaves behind when one of its waits ran out, set from the host: the next call on the device raises, whichever way it comes,
    and the one after that is an ordinary call again."""
    from sgl_kernel.quantization import bitnet_gemm, bitnet_gemv
    from test_gpu_engine import small_cfg
    from wf_bitnet import ops
    from wf_bitnet._lib import WfError, lib
    from wf_bitnet.engine import Engine
    from wf_bitnet.synth import make_weights
    word = lib().wf_wait_word()
    assert word and word[0] == 0
    n, k, m = 512, 640, 48
    rng = np.random.default_rng(4)
    code = rng.integers(0, 3, size=(n, k // 128, 4, 32)).astype(np.uint8)
    pi = cu((code[:, :, 0] << 6 | code[:, :, 1] << 4 | code[:, :, 2] << 2 | code[:, :, 3]).reshape(n, k // 4))
    q = torch.from_numpy(rng.integers(-128, 128, size=(m, k)).astype(np.int8)).cuda()
    x = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    g, f = torch.ones(n, device="cuda", dtype=torch.bfloat16), cu(np.full((k, n // 4), 0x55, np.uint8))
    cfg = small_cfg()
    engine = Engine(cfg)
    engine.load_weights(make_weights(cfg, seed=1234))
    calls = [lambda: bitnet_gemm(pi, q, 0.5), lambda: bitnet_gemv(pi, q[0], 0.5), lambda: ops.ternary_linear(pi, n, k, q, layout="i2s", mode="i32_plus1"),
             lambda: torch.ops.sgl_kernel.bitnet_mlp_forward_cpu(x, pi, pi, f, 0.1, 0.1, 0.1, g, 1e-5), lambda: engine.decode([5])]
    for i, call in enumerate(calls):
        call()
        torch.cuda.synchronize()
        word[0] = 4
        with pytest.raises(WfError, match="ran out"):
            call()
        assert word[0] == 0, i
        call()
    torch.cuda.synchronize()
    assert torch.equal(calls[0]().cpu(), torch.from_numpy(O.gemm_i32_fast(pi.cpu().numpy(), q.cpu().numpy(), 0).astype(np.float32) * np.float32(0.5)))
    engine.close()


def test_the_first_product_of_a_process_may_be_captured():
    """A process whose first product, one on CTA pairs, lies in a graph capture that allows nothing unsafe to any thread."""
    import subprocess
    import sys
    code = """
import torch, sgl_kernel
from sgl_kernel.quantization import bitnet_gemm
w = torch.randint(0, 256, (14336, 1024), device="cuda", dtype=torch.uint8) & 0xAA
x = torch.randint(-127, 128, (48, 4096), device="cuda", dtype=torch.int8)
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g, capture_error_mode="global"):
    y = bitnet_gemm(w, x, 0.5)
g.replay()
torch.cuda.synchronize()
assert torch.equal(y, bitnet_gemm(w, x, 0.5)) and float(y.abs().sum()) > 0
print("equal")
"""
    from conftest import PKG
    r = subprocess.run([sys.executable, "-c", code], cwd=str(PKG), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "equal", r.stderr[-2000:]


@pytest.mark.parametrize("nkm", [(256, 128, 40), (6912, 2560, 300)])
def test_tc_pairs_subtract_whole_sums(nkm):
    """Sums of activations beyond 2^24, which K above 131072 or a caller's own sums bring: subtracted as the whole numbers that they are."""
    from wf_bitnet import ops
    n, k, m = nkm
    rng = np.random.default_rng(k)
    q = torch.from_numpy(rng.integers(-128, 128, size=(m, k)).astype(np.int8)).cuda()
    w = cu(rng.integers(0, 256, size=(n, k // 4)).astype(np.uint8) & 0xAA)
    rs = torch.from_numpy(rng.integers(-(1 << 30), 1 << 30, size=m).astype(np.int32) | 1).cuda()
    a, b = (ops.ternary_linear(w, n, k, q, layout="i2s", mode="i32", rowsum=rs, algo=x) for x in (3, 2))
    assert torch.equal(a, b)
