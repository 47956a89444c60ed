"""The sequence engine's matrix product on tensor cores: CTA pairs (token tiles that are no whole tile, rows that leave the second CTA empty, several rounds
of tiles) and the few-row form (row tiles short of 16, K that is no multiple of its steps, each split of the work).

Tolerance: float sums of K bf16 products in another order, a few times 2^-24 sqrt(K) of the operands' unit scale; 2e-5 covers K = 7000 on the tcgen05 sum."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def product(A, B, algo, c_f32=True):
    from wf_bitnet._lib import seq_check, seq_lib
    (M, K), N = A.shape, B.shape[0]
    C = torch.full((M, N), float("nan"), dtype=torch.float32 if c_f32 else torch.bfloat16, device="cuda")
    seq_check(seq_lib().wf_seq_op_gemm(1, A.data_ptr(), 0, K, B.data_ptr(), K, C.data_ptr(), 1 if c_f32 else 0, N, M, N, K, None, 0, 1, algo,
                                       torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return C


def operands(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + 7 * K)
    return torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16), (torch.randn(N, K, device="cuda", generator=g) / math.sqrt(K)).to(torch.bfloat16)


@pytest.mark.parametrize("M,N,K", [(17, 8, 8), (33, 129, 72), (255, 257, 64), (257, 255, 200), (1000, 130, 1032), (530, 2561, 320), (2049, 1024, 6912), (3000, 5000, 64)])
def test_pair_product(M, N, K):
    A, B = operands(M, N, K)
    want = A.double() @ B.double().T
    assert (product(A, B, 3).double() - want).abs().max() < 2e-5 * (1 + want.abs().max())
    assert (product(A, B, 3, c_f32=False).double() - want).abs().max() < 2.0 ** -8 * (1 + want.abs().max())


@pytest.mark.parametrize("M", [1, 3, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(1, 8), (15, 40), (17, 72), (1000, 2304), (2560, 6912), (4737, 264), (9473, 1000), (30000, 136)])
def test_few_rows(M, N, K):
    A, B = operands(M, N, K)
    want = A.double() @ B.double().T
    assert (product(A, B, 5).double() - want).abs().max() < 5e-6 * (1 + want.abs().max())
    assert (product(A, B, 5, c_f32=False).double() - want).abs().max() < 2.0 ** -8 * (1 + want.abs().max())


@pytest.mark.parametrize("M", [1, 8])
@pytest.mark.parametrize("K", [8, 520])
@pytest.mark.parametrize("tiles", [(2, 1), (4, 0), (4, 1), (8, 1), (12, 0), (12, 1)])
def test_few_rows_where_the_tiles_of_a_block_change(M, K, tiles):
    """Blocks of one tile of 16 rows or of two, by the rounds that they make on four blocks an SM: widths on both sides of each change, the last tile short of 16."""
    per_sm, more = tiles
    N = 16 * per_sm * torch.cuda.get_device_properties(0).multi_processor_count + (3 if more else 0)
    A, B = operands(M, N, K)
    want = A.double() @ B.double().T
    assert (product(A, B, 5).double() - want).abs().max() < 5e-6 * (1 + want.abs().max())


@pytest.mark.parametrize("M", [1, 8])
@pytest.mark.parametrize("K", [1024, 2560, 6912, 28672])
def test_few_rows_are_as_close_as_multiply_adds(M, K):
    """Against 64 bits the matrix-unit form of up to 8 rows is no further off than the multiply-add form.  Four samples of 1024 sums or more leave each 2-norm
    uncertain by about 1 %."""
    off = [0., 0.]
    for i in range(4):
        g = torch.Generator(device="cuda").manual_seed(1000 * i + K + M)
        A = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
        B = (torch.randn(1024, K, device="cuda", generator=g) / math.sqrt(K)).to(torch.bfloat16)
        want = A.double() @ B.double().T
        off[0] += float((product(A, B, 5).double() - want).norm() / want.norm())
        off[1] += float((product(A, B, 4).double() - want).norm() / want.norm())
    assert off[0] < 1.03 * off[1], off


def test_the_row_limit_of_the_tcgen05_form_holds_below_17(tmp_path):
    """WF_SEQ_TC_MIN = 9: products of 9 to 16 rows are the tcgen05 form's, bit for bit; by default the few-row form's."""
    import os
    import subprocess
    import sys
    from pathlib import Path
    here = Path(__file__).resolve().parent
    code = ("import torch, test_gpu_seq_gemm as t\n"
            "for m, n, k in ((9, 300, 1000), (16, 2560, 2560)):\n"
            "    A, B = t.operands(m, n, k)\n"
            "    print(int(torch.equal(t.product(A, B, 0), t.product(A, B, 3))), int(torch.equal(t.product(A, B, 0), t.product(A, B, 5))))\n")
    for limit, want in (("9", "1 0"), ("17", "0 1")):
        env = dict(os.environ, WF_SEQ_TC_MIN=limit, PYTHONPATH=f"{here}:{here.parent / 'wrinklefree-inference-engine_b200'}")
        r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        assert r.stdout.split("\n")[:2] == [want, want], r.stdout


@pytest.mark.parametrize("ff", [16, 44, 48, 144, 272])
@pytest.mark.parametrize("design", ["tutizen", "nukezen"])
def test_gated_unit_in_the_product(design, ff):
    """Feed-forwards whose activation is formed where the product stores its results: few rows, gate and up rows in blocks of 8; many rows, blocks of 16, a CTA's
    last blocks missing, token tiles that are not whole (44 has no such blocks and keeps the separate kernel there); both activations, against the sum in 64 bits on the same bf16 operands.

    Tolerance: the hidden values and the output's operands are rounded to bf16 (2^-9 each); 1e-2 of a row's size is two and a half times that."""
    import numpy as np
    import importlib
    t = importlib.import_module("test_gpu_" + design)
    W = 64
    if design == "tutizen":
        cfg = t.config([t.with_ff(t.attn(), t.dense(ff=ff))], width=W)
    else:
        cfg = t.config([t.par(ff=ff)], width=W)
    w = {k: torch.from_numpy(np.asarray(v, np.float32)).to(torch.bfloat16).float().numpy() for k, v in t.make_weights(cfg if design == "tutizen" else (cfg, {}), ff).items()}
    m = t.build(cfg, w, "bfloat16", max_tokens=512, max_step_tokens=384)
    g = {k[len("l0.mlp."):]: torch.from_numpy(v).double() for k, v in w.items() if k.startswith("l0.mlp.")}
    for n in (1, 7, 16, 17, 33, 300):
        x = torch.randn(n, W, generator=torch.Generator().manual_seed(n + ff)).to(torch.bfloat16).double() * 2
        gate, up = x @ g["gate"].T, x @ g["up"].T
        if design == "tutizen":
            lim = cfg["layers"][0]["mlp"]["limit"]
            gate, up = gate.clamp(max=lim), up.clamp(-lim, lim)
            h = gate * torch.sigmoid(1.702 * gate) * (up + 1)
        else:
            h = torch.nn.functional.gelu(gate, approximate="tanh") * up
        want = (h @ g["down"].T).numpy()
        slot = m.admit()
        got = m.engine.run_part(0, 3, [slot], [n], x.float().numpy())
        m.release(slot)
        err = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
        assert err.max() < 1e-2, (n, err.max())
    m.close()
