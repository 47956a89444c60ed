"""The 16-token form of the matrix-state recurrences against the oracles, in float32, where it has to be asked for: every length around its chunks, long portions in parallel segments,
portions behind carried states, several sequences side by side, key sizes that do not fill a thread's rows, value sizes that do not fill a block.

Tolerance: float32 sums over at most a few hundred terms of order one in another order, relative to a row's RMS; the delta rule's correction solves
a 16 x 16 triangular system per chunk, whose condition the unit-length keys and beta < 1 keep below a few tens: 2e-4, as for the token form."""
import numpy as np
import pytest
import torch

import fivedra_oracle as FO
import nukezen_oracle as NO

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def sixteen_token_form(monkeypatch):
    monkeypatch.setenv("WF_SEQ_CHUNK", "1")        # float32 engines keep the token form by themselves


CUTS = [([70], [[70]]), ([33, 100], [[33, 100]]), ([90, 64], [[32, 0], [15, 47], [43, 16], [0, 1]]), ([47], [[47]]), ([545, 140], [[21, 0], [524, 140]])]
EPS = 1e-5


def check(cfg, weights, shapes, wants, lens, cuts, W, max_tokens=800, step=672):
    from wf_bitnet import registry
    cls = registry.resolve(cfg)
    extra = {"shapes": shapes} if getattr(cls, "reads_shapes", False) else {}
    m = cls(cfg, dtype="float32", max_tokens=max_tokens, slots=4, page_size=16, max_step_tokens=step, **extra)
    m.load_weights((k, v.numpy(), "F32") for k, v in weights.items())
    g = np.random.default_rng(sum(lens))
    rows = [g.standard_normal((n, W)).astype(np.float32) for n in lens]
    slots, fed = [m.admit() for _ in rows], [0] * len(rows)
    want = [wants(torch.from_numpy(r).double()).numpy() for r in rows]
    for step in cuts:
        act = [i for i, c in enumerate(step) if c]
        got = m.engine.run_part(0, 2, [slots[i] for i in act], [step[i] for i in act], np.concatenate([rows[i][fed[i]:fed[i] + step[i]] for i in act]))
        w = np.concatenate([want[i][fed[i]:fed[i] + step[i]] for i in act])
        err = np.sqrt(((got - w) ** 2).mean(-1)) / np.sqrt((w ** 2).mean(-1))
        assert err.max() < 2e-4, (step, int(err.argmax()), err.max())
        for i in act:
            fed[i] += step[i]
    m.close()


def d64(w, p):
    return {k[len(p):]: v.double() for k, v in w.items() if k.startswith(p)}


@pytest.mark.parametrize("lens,cuts", CUTS)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(4, 2, 128, 128), (2, 2, 36, 20), (40, 20, 64, 96), (3, 1, 68, 33)])
def test_delta_rule_with_a_decay_per_row(heads, kv_heads, dim, vdim, lens, cuts):
    W = 40
    m = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": vdim, "conv": 4}
    cfg = {"architecture": "Nukezen", "vocab": 31, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": EPS}, "layers": [{"type": "channel_delta", "mixer": m, "mlp": None}]}
    w = NO.random_weights(cfg, 1, {0: {"rank_a": 8, "rank_g": 8}})
    check(cfg, w, {"l0.mix.a1": (8, W), "l0.mix.g1": (8, W)}, lambda x: NO.channel_delta(x, d64(w, "l0.mix."), "", m, EPS), lens, cuts, W)


@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(60, 20, 64, 97), (64, 16, 64, 97), (40, 20, 100, 130), (160, 20, 36, 20)])
def test_delta_rule_of_many_heads(heads, kv_heads, dim, vdim):
    """Enough (sequence, head, 16 columns) tiles that a block takes two of them (not with 60 heads), the last one of an odd count alone."""
    W = 40
    m = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": vdim, "conv": 4}
    cfg = {"architecture": "Nukezen", "vocab": 31, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": EPS}, "layers": [{"type": "channel_delta", "mixer": m, "mlp": None}]}
    w = NO.random_weights(cfg, 1, {0: {"rank_a": 8, "rank_g": 8}})
    check(cfg, w, {"l0.mix.a1": (8, W), "l0.mix.g1": (8, W)}, lambda x: NO.channel_delta(x, d64(w, "l0.mix."), "", m, EPS), [90, 64], [[32, 17], [15, 47], [43, 0]], W)


@pytest.mark.parametrize("lens", [[200, 330], [330, 200], [60, 400, 90]])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(20, 10, 128, 128), (12, 12, 64, 97), (30, 10, 68, 33)])
def test_delta_rule_of_portions_of_unequal_length(heads, kv_heads, dim, vdim, lens):
    """The longest portion in blocks of one column tile, wherever it stands, and the others in blocks of two (an odd last one), each behind a carried state."""
    W = 40
    m = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": vdim, "conv": 4}
    cfg = {"architecture": "Nukezen", "vocab": 31, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": EPS}, "layers": [{"type": "channel_delta", "mixer": m, "mlp": None}]}
    w = NO.random_weights(cfg, 1, {0: {"rank_a": 8, "rank_g": 8}})
    check(cfg, w, {"l0.mix.a1": (8, W), "l0.mix.g1": (8, W)}, lambda x: NO.channel_delta(x, d64(w, "l0.mix."), "", m, EPS), lens, [[3] * len(lens), [n - 3 for n in lens]], W, 1000)


@pytest.mark.parametrize("conv", [2, 3])
def test_convolutions_of_two_and_three_taps_over_many_tokens(conv):
    """Enough tokens x channels (6400) that a thread of the convolution takes four tokens one after another: portions that begin and end inside such a run, behind a carried
    state of one and two inputs, and a portion of one token."""
    W = 40
    m = {"heads": 40, "kv_heads": 20, "dim": 64, "vdim": 96, "conv": conv}
    cfg = {"architecture": "Nukezen", "vocab": 31, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": EPS}, "layers": [{"type": "channel_delta", "mixer": m, "mlp": None}]}
    w = NO.random_weights(cfg, 1, {0: {"rank_a": 8, "rank_g": 8}})
    check(cfg, w, {"l0.mix.a1": (8, W), "l0.mix.g1": (8, W)}, lambda x: NO.channel_delta(x, d64(w, "l0.mix."), "", m, EPS), [391, 203], [[190, 1], [1, 199], [200, 3]], W)


@pytest.mark.parametrize("lens,cuts", CUTS)
@pytest.mark.parametrize("heads,groups,state,vdim", [(4, 2, 128, 64), (6, 3, 20, 12), (80, 5, 64, 64)])
def test_state_space(heads, groups, state, vdim, lens, cuts):
    W = 40
    left = {"heads": 2, "kv_heads": 1, "dim": 8, "vdim": 8, "scale": 0.3, "mask": {"size": 8}, "rot": {"dims": 8, "base": 10000.0}}
    right = {"heads": heads, "vdim": vdim, "state": state, "groups": groups, "conv": 4, "norm_groups": groups}
    cfg = {"architecture": "Nukezen", "vocab": 31, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": EPS},
           "layers": [{"type": "parallel", "mixer": {"left": left, "left_scale": 0.0, "right": right, "right_scale": 1.0}, "mlp": None}]}
    w = NO.random_weights(cfg, 2)
    check(cfg, w, {}, lambda x: NO.state_space(x, d64(w, "l0.mix.right."), "", right, EPS), lens, cuts, W)


@pytest.mark.parametrize("lens,cuts", CUTS)
@pytest.mark.parametrize("heads,dim,vdim", [(4, 128, 128), (3, 24, 15), (150, 20, 36)])
def test_matrix_memory(heads, dim, vdim, lens, cuts):
    W = 40
    left = {"heads": 2, "kv_heads": 1, "dim": 8, "vdim": 8, "scale": 0.3, "mask": {"size": 8}, "bias_max": 16}
    right = {"heads": heads, "dim": dim, "vdim": vdim, "gate_cap": 15.0}
    cfg = {"architecture": "Fivedra", "vocab": 31, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": EPS},
           "layers": [{"type": "parallel", "mixer": {"left": left, "left_scale": 0.0, "right": right, "right_scale": 1.0}, "mlp": None}]}
    w = FO.random_weights(cfg, 3)
    check(cfg, w, {"l0.mix.left.rel": (8, 2)}, lambda x: FO.matrix_memory(x, d64(w, "l0.mix.right."), "", right, EPS), lens, cuts, W)


# long portions, of which some sizes of heads take some in segments of 128 tokens all at once
@pytest.mark.parametrize("lens,cuts", [([512], [[512]]), ([670, 513], [[30, 513], [640, 0]]), ([639], [[639]])])
@pytest.mark.parametrize("kind,heads,groups,dim,vdim", [("ssd", 4, 2, 128, 64), ("ssd", 6, 3, 20, 12), ("ssd", 8, 1, 64, 68), ("memory", 2, 2, 128, 128), ("memory", 3, 3, 24, 15)])
def test_segments(kind, heads, groups, dim, vdim, lens, cuts):
    check_plain(kind, heads, groups, dim, vdim, lens, cuts)


# Whole segments, a last one of one token and of one less than a whole one, a carried state, a sequence of less than a segment beside them; key sizes that leave rows of a warp over,
# value sizes below, at and beyond 64 columns, several heads on a key head and one
@pytest.mark.parametrize("kind,heads,groups,dim,vdim,lens,cuts", [
    *((*k, *c) for k in (("ssd", 8, 2, 128, 64), ("ssd", 6, 3, 20, 12), ("ssd", 8, 1, 64, 68), ("memory", 3, 3, 24, 15), ("memory", 14, 14, 128, 128))
      for c in (([799, 70], [[30, 0], [769, 70]]), ([767, 31], [[767, 31]]), ([768, 1], [[768, 1]]))),
    ("ssd", 32, 1, 64, 68, [512], [[512]]), ("ssd", 24, 2, 68, 33, [640, 513], [[640, 513]]), ("ssd", 32, 1, 64, 68, [540, 639], [[28, 0], [512, 639]])])
def test_portions_taken_in_segments(kind, heads, groups, dim, vdim, lens, cuts):
    from wf_bitnet import _lib
    assert _lib.seq_lib().wf_seq_in_segments(heads, groups, dim, vdim, kind == "memory", sum(c > 0 for c in cuts[-1]), sum(cuts[-1]), max(cuts[-1]))
    check_plain(kind, heads, groups, dim, vdim, lens, cuts)


def check_plain(kind, heads, groups, dim, vdim, lens, cuts):
    W = 40
    left = {"heads": 2, "kv_heads": 1, "dim": 8, "vdim": 8, "scale": 0.3, "mask": {"size": 8}}
    if kind == "ssd":
        left["rot"] = {"dims": 8, "base": 10000.0}
        right = {"heads": heads, "vdim": vdim, "state": dim, "groups": groups, "conv": 4, "norm_groups": groups}
    else:
        left["bias_max"] = 16
        right = {"heads": heads, "dim": dim, "vdim": vdim, "gate_cap": 15.0}
    cfg = {"architecture": "Nukezen" if kind == "ssd" else "Fivedra", "vocab": 31, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": EPS},
           "layers": [{"type": "parallel", "mixer": {"left": left, "left_scale": 0.0, "right": right, "right_scale": 1.0}, "mlp": None}]}
    w = (NO if kind == "ssd" else FO).random_weights(cfg, 4)
    oracle = (lambda x: NO.state_space(x, d64(w, "l0.mix.right."), "", right, EPS)) if kind == "ssd" else (lambda x: FO.matrix_memory(x, d64(w, "l0.mix.right."), "", right, EPS))
    check(cfg, w, {} if kind == "ssd" else {"l0.mix.left.rel": (8, 2)}, oracle, lens, cuts, W, 1400, 1184)


# ---- numbers that are not finite: long portions (the 16-token form, and its parallel segments where the recurrence is plain) against the same rows in portions of 31 tokens (token by token)
def nonfinite_layer(kind):
    W = 40
    if kind == "delta":
        m = {"heads": 4, "kv_heads": 2, "dim": 64, "vdim": 32, "conv": 4}
        cfg = {"architecture": "Nukezen", "vocab": 31, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": EPS}, "layers": [{"type": "channel_delta", "mixer": m, "mlp": None}]}
        return cfg, NO.random_weights(cfg, 1, {0: {"rank_a": 8, "rank_g": 8}}), {"l0.mix.a1": (8, W), "l0.mix.g1": (8, W)}, W
    left = {"heads": 2, "kv_heads": 1, "dim": 8, "vdim": 8, "scale": 0.3, "mask": {"size": 8}}
    if kind == "state_space":
        left["rot"] = {"dims": 8, "base": 10000.0}
        right = {"heads": 4, "vdim": 32, "state": 64, "groups": 2, "conv": 4, "norm_groups": 2}
        arch, make, shapes = "Nukezen", lambda c: NO.random_weights(c, 2), {}
    else:
        left["bias_max"] = 16
        right = {"heads": 4, "dim": 64, "vdim": 32, "gate_cap": 15.0}
        arch, make, shapes = "Fivedra", lambda c: FO.random_weights(c, 3), {"l0.mix.left.rel": (8, 2)}
    cfg = {"architecture": arch, "vocab": 31, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": EPS},
           "layers": [{"type": "parallel", "mixer": {"left": left, "left_scale": 0.0, "right": right, "right_scale": 1.0}, "mlp": None}]}
    return cfg, make(cfg), shapes, W


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), 3e38, 1e13])
@pytest.mark.parametrize("at", [0, 37, 530, 745])
@pytest.mark.parametrize("kind", ["state_space", "memory"])
def test_numbers_that_are_not_finite_in_segments(kind, at, bad, monkeypatch):
    """The same for a long portion and a short one beside it in segments: such a number in one of them (from row 740 on the short one's) leaves the other as it is."""
    from wf_bitnet import _lib, registry
    assert _lib.seq_lib().wf_seq_in_segments(4, 2 if kind == "state_space" else 4, 64, 32, kind == "memory", 2, 800, 740)
    monkeypatch.setenv("WF_SEQ_ATTN_MMA", "0")
    cfg, weights, shapes, W = nonfinite_layer(kind)
    cls = registry.resolve(cfg)
    extra = {"shapes": shapes} if getattr(cls, "reads_shapes", False) else {}
    m = cls(cfg, dtype="bfloat16", max_tokens=2000, slots=4, page_size=16, max_step_tokens=800, **extra)
    m.load_weights((k, v.numpy(), "F32") for k, v in weights.items())
    g = np.random.default_rng(8)
    rows = torch.from_numpy(g.standard_normal((900, W)).astype(np.float32)).to(torch.bfloat16).float().numpy()
    rows[at, 3] = bad
    first, second = np.r_[0:740, 800:850], np.r_[740:800, 850:900]         # what each sequence is fed: a portion of the first step, then 50 rows
    a, b, c, d = (m.admit() for _ in range(4))
    whole = np.empty((900, W), np.float32)
    whole[:800], whole[800:] = m.engine.run_part(0, 2, [a, b], [740, 60], rows[:800]), m.engine.run_part(0, 2, [a, b], [50, 50], rows[800:])
    pieces = np.empty_like(whole)
    for slot, idx in ((c, first), (d, second)):
        pieces[idx] = np.concatenate([m.engine.run_part(0, 2, [slot], [len(idx[t:t + 31])], rows[idx[t:t + 31]]) for t in range(0, len(idx), 31)])
    m.close()
    ok, want = np.isfinite(whole).all(-1), np.isfinite(pieces).all(-1)
    assert np.array_equal(ok, want), (np.flatnonzero(ok != want), ok.sum(), want.sum())
    hit = first if at < 740 else second
    clean = np.r_[second if at < 740 else first, hit[hit < at]]
    assert want[clean].all()
    x, y = whole[clean], pieces[clean]
    assert (np.sqrt(((x - y) ** 2).mean(-1)) / np.sqrt((y ** 2).mean(-1))).max() < 2e-2          # two bf16 roundings of the same float values, and the products around them


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), 3e38, 1e13])
@pytest.mark.parametrize("at", [0, 37, 530])
@pytest.mark.parametrize("kind", ["delta", "state_space", "memory"])
def test_numbers_that_are_not_finite(kind, at, bad, monkeypatch):
    """A token whose row holds a NaN, an infinity or a number that overflows on the way: the same output rows are finite as token by token, in the portion and in the next one."""
    from wf_bitnet import registry
    monkeypatch.setenv("WF_SEQ_ATTN_MMA", "0")         # the pair's other mixer keeps such numbers to the rows that see them
    cfg, weights, shapes, W = nonfinite_layer(kind)
    cls = registry.resolve(cfg)
    extra = {"shapes": shapes} if getattr(cls, "reads_shapes", False) else {}
    m = cls(cfg, dtype="bfloat16", max_tokens=1600, slots=4, page_size=16, max_step_tokens=600, **extra)
    m.load_weights((k, v.numpy(), "F32") for k, v in weights.items())
    g = np.random.default_rng(7)
    rows = torch.from_numpy(g.standard_normal((700, W)).astype(np.float32)).to(torch.bfloat16).float().numpy()
    rows[at, 3] = bad
    a, b = m.admit(), m.admit()
    whole = np.concatenate([m.engine.run_part(0, 2, [a], [n], rows[t:t + n]) for t, n in ((0, 600), (600, 100))])
    pieces = np.concatenate([m.engine.run_part(0, 2, [b], [min(31, 700 - t)], rows[t:t + 31]) for t in range(0, 700, 31)])
    m.close()
    ok, want = np.isfinite(whole).all(-1), np.isfinite(pieces).all(-1)
    assert np.array_equal(ok, want), (np.flatnonzero(ok != want), ok.sum(), want.sum())
    assert want[:at].all()
    if want[:at].any():
        x, y = whole[:at], pieces[:at]
        err = np.sqrt(((x - y) ** 2).mean(-1)) / np.sqrt((y ** 2).mean(-1))
        assert err.max() < 2e-2          # two bf16 roundings of the same float values, and the products around them


def test_float32_engines_keep_the_token_form(monkeypatch):
    """By default a float32 engine gives the bits of plain multiply-adds token by token, a bf16 engine those of the 16-token form."""
    from wf_bitnet import registry
    cfg, weights, shapes, W = nonfinite_layer("delta")
    rows = np.random.default_rng(1).standard_normal((200, W)).astype(np.float32)

    def run(dtype, form):
        monkeypatch.delenv("WF_SEQ_CHUNK") if form is None else monkeypatch.setenv("WF_SEQ_CHUNK", form)
        cls = registry.resolve(cfg)
        extra = {"shapes": shapes} if getattr(cls, "reads_shapes", False) else {}
        m = cls(cfg, dtype=dtype, max_tokens=400, slots=2, page_size=16, max_step_tokens=256, **extra)
        m.load_weights((k, v.numpy(), "F32") for k, v in weights.items())
        out = m.engine.run_part(0, 2, [m.admit()], [200], rows)
        m.close()
        monkeypatch.setenv("WF_SEQ_CHUNK", "1")
        return out
    assert np.array_equal(run("float32", None), run("float32", "0")) and not np.array_equal(run("float32", "0"), run("float32", "1"))
    assert np.array_equal(run("bfloat16", None), run("bfloat16", "1"))
