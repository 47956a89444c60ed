"""An engine on a device that is nearly full: what only the faster prompt forms need is left out, and the rest works as without them."""
import numpy as np
import pytest
import torch

import fivedra_oracle as FO

pytestmark = pytest.mark.gpu


def test_the_workspaces_of_the_faster_forms_are_not_required(monkeypatch):
    from wf_bitnet import registry
    W = 64
    m = {"heads": 20, "dim": 96, "rot_dim": 32, "vdim": 128, "kv_rank": 512, "q_rank": 48, "scale": 128 ** -0.5,
         "rot": {"dims": 32, "base": 10000.0, "scaling": {"factor": 4.0, "original": 256, "fast": 32.0, "slow": 1.0}}}
    cfg = {"architecture": "Fivedra", "vocab": 31, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5},
           "layers": [{"type": "latent_attention", "mixer": m, "mlp": None}]}
    weights = FO.random_weights(cfg, 1)
    rows = np.random.default_rng(2).standard_normal((900, W)).astype(np.float32)

    def build():
        cls = registry.resolve(cfg)
        extra = {"shapes": {}} if getattr(cls, "reads_shapes", False) else {}
        e = cls(cfg, dtype="bfloat16", max_tokens=32768, slots=2, page_size=16, max_step_tokens=8192, **extra)
        e.load_weights((k, v.numpy(), "F32") for k, v in weights.items())
        return e

    def run(e):
        out = e.engine.run_part(0, 2, [e.admit()], [900], rows)
        size = e.engine.device_bytes()
        e.close()
        return out, size
    monkeypatch.setenv("WF_SEQ_ATTN_MMA", "2")
    plain, small = run(build())
    monkeypatch.delenv("WF_SEQ_ATTN_MMA")
    _, full = run(build())
    assert full > small + (200 << 20)
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    held = torch.empty(free - small - (256 << 20), dtype=torch.uint8, device="cuda")
    try:
        tight, size = run(build())
    finally:
        del held
        torch.cuda.empty_cache()
    assert size == small and np.array_equal(tight, plain)


@pytest.mark.parametrize("vocab,wants", [(4099, (1, 64, 65, 180)), (65536, (1, 2, 8, 11))])
def test_logits_reach_pageable_memory_as_they_reach_pinned(vocab, wants):
    """One piece, whole pieces, a part of a piece, more pieces than are in flight at once (512 KB each, four at once): equal to one copy into pinned memory."""
    from wf_bitnet._lib import seq_check, seq_lib
    from test_gpu_tutizen import attn, build, config, make_weights, with_ff, dense
    cfg = config([with_ff(attn(), dense())], vocab=vocab)
    m = build(cfg, make_weights(cfg, 3), "bfloat16", max_tokens=1024, slots=2, page_size=16, max_step_tokens=256)
    rng = np.random.default_rng(vocab)
    for n in wants:
        toks = rng.integers(0, vocab, max(n, 2)).astype(np.int32)
        rows = np.sort(rng.choice(toks.size, n, replace=False)).astype(np.int32)
        slot = m.admit()
        got = m.step([slot], [toks.size], toks, rows)
        m.release(slot)
        pinned = torch.full((n, vocab), float("nan")).pin_memory()
        slot = m.admit()
        s, c = np.array([slot], np.int32), np.array([toks.size], np.int32)
        seq_check(seq_lib().wf_seq_step(m.engine._h, 1, s.ctypes.data, c.ctypes.data, toks.ctypes.data, n, rows.ctypes.data, pinned.data_ptr()))
        m.release(slot)
        assert np.isfinite(got).all() and np.array_equal(got, pinned.numpy()), n
    m.close()


def test_a_large_block_table_is_not_page_locked():
    """32 slots x 16,384 pages, a table of 2 MB: the same tokens as with a small table, over steps that add pages and that do not."""
    from test_gpu_tutizen import attn, build, config, make_weights, with_ff, dense
    cfg = config([with_ff(attn(), dense())], vocab=70)
    w = make_weights(cfg, 3)
    outs = []
    for pages in (64, 16384):
        m = build(cfg, w, "bfloat16", max_tokens=pages * 4, slots=32, page_size=4, max_step_tokens=64)
        assert m.engine.free_pages() == pages
        a, b = m.admit(), m.admit()
        rng = np.random.default_rng(1)
        got = []
        for counts in ([13, 5], [1, 1], [2, 1], [1, 1], [30, 9]):
            got.append(m.step([a, b], counts, rng.integers(0, 70, sum(counts)).astype(np.int32), np.arange(sum(counts), dtype=np.int32)))
        m.release(a)
        c = m.admit()
        got.append(m.step([b, c], [3, 20], rng.integers(0, 70, 23).astype(np.int32), np.arange(23, dtype=np.int32)))
        outs.append(np.concatenate(got))
        m.close()
    assert np.isfinite(outs[0]).all() and np.array_equal(outs[0], outs[1])
