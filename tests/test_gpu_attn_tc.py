"""Prompt attention on tcgen05 against the plain oracles: edges of its 128-key and 128-row tiles, head groupings that leave rows unused, head sizes
below a swizzle block, page sizes from 8 keys to more than a tile, windows, sequences side by side, portions behind cached keys.

Tolerance: the bf16 engine rounds the mixer's input products' operands, q, k, v, the output rows and (latent form) the weights and expanded keys to
2^-9 relative; a handful of independent roundings over random signs stay below 1e-2 of a row's RMS, and 2e-2 leaves a factor of two."""
import numpy as np
import pytest
import torch

import fivedra_oracle as FO
import nukezen_oracle as NO
import tutizen_oracle as TO

pytestmark = pytest.mark.gpu
TOL = 2e-2


def build(cfg, weights, page_size, shapes=None):
    from wf_bitnet import registry
    cls = registry.resolve(cfg)
    extra = {"shapes": shapes} if getattr(cls, "reads_shapes", False) else {}
    m = cls(cfg, dtype="bfloat16", max_tokens=2048, slots=4, page_size=page_size, max_step_tokens=700, **extra)
    m.load_weights((k, v.numpy(), "F32") for k, v in weights.items())
    return m


def check(m, rows, cuts, wants, W):
    """rows: one array per sequence; cuts: the steps, each the tokens every sequence brings.  Every output row against wants."""
    slots = [m.admit() for _ in rows]
    fed = [0] * len(rows)
    for step in cuts:
        act = [i for i, c in enumerate(step) if c]
        x = np.concatenate([rows[i][fed[i]:fed[i] + step[i]] for i in act])
        got = m.engine.run_part(0, 2, [slots[i] for i in act], [step[i] for i in act], x)
        want = np.concatenate([wants[i][fed[i]:fed[i] + step[i]] for i in act])
        err = np.sqrt(((got - want) ** 2).mean(-1)) / np.sqrt((want ** 2).mean(-1))
        assert err.max() < TOL, (step, int(err.argmax()), err.max())
        for i in act:
            fed[i] += step[i]
    for s in slots:
        m.release(s)


def inputs(lens, W, seed):
    g = np.random.default_rng(seed)
    return [torch.from_numpy(g.standard_normal((n, W)).astype(np.float32)).to(torch.bfloat16).float().numpy() for n in lens]


def d64(weights, prefix):
    return {k[len(prefix):]: v.double() for k, v in weights.items() if k.startswith(prefix)}


# (the form takes steps in which some sequence reaches more than 256 keys)
CUTS = {"whole": ([520, 129], [[520, 129]]), "portions": ([520, 129], [[300, 2], [2, 0], [82, 126], [136, 1]]), "tiles": ([512, 128], [[384, 128], [128, 0]]), "start": ([257, 1], [[257, 1]])}


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,page", [(4, 4, 128, 128, 16), (8, 2, 128, 64, 8), (5, 1, 72, 128, 256), (6, 2, 64, 40, 128), (16, 1, 8, 8, 16)])
@pytest.mark.parametrize("cut", list(CUTS))
def test_penalty_and_head_gates(heads, kv_heads, dim, vdim, page, cut):
    W = 64
    m = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": vdim, "scale": dim ** -0.5}
    cfg = {"architecture": "Tutizen", "vocab": 31, "width": W, "norm": {"eps": 1e-5}, "residual_mult": 1.0, "layers": [{"type": "attention", "mixer": m, "mlp": None}]}
    w = TO.random_weights(cfg, heads + dim)
    lens, cuts = CUTS[cut]
    rows = inputs(lens, W, 3)
    P = d64(w, "l0.mix.")
    wants = [TO.attention(torch.from_numpy(r).double(), P, m, 1e-5)[0].numpy() for r in rows]
    model = build(cfg, w, page)
    check(model, rows, cuts, wants, W)
    model.close()


@pytest.mark.parametrize("window", [257, 300, 384, 385, 1000])
@pytest.mark.parametrize("cut", ["whole", "portions"])
def test_window_rotation_and_element_gates(window, cut):
    W = 64
    left = {"heads": 6, "kv_heads": 2, "dim": 64, "vdim": 64, "scale": 0.125, "mask": {"size": window}, "rot": {"dims": 32, "base": 10000.0}}
    right = {"heads": 2, "vdim": 8, "state": 8, "groups": 1, "conv": 4, "norm_groups": 1}
    cfg = {"architecture": "Nukezen", "vocab": 31, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5},
           "layers": [{"type": "parallel", "mixer": {"left": left, "left_scale": 1.0, "right": right, "right_scale": 0.0}, "mlp": None}]}
    w = NO.random_weights(cfg, window)
    lens, cuts = CUTS[cut]
    rows = inputs(lens, W, 5)
    P = d64(w, "l0.mix.left.")
    wants = [NO.window_attention(torch.from_numpy(r).double(), P, "", left, 1e-5).numpy() for r in rows]
    model = build(cfg, w, 16, {})
    check(model, rows, cuts, wants, W)
    model.close()


@pytest.mark.parametrize("heads,dim,rot,vdim,rank", [(20, 96, 32, 128, 512), (8, 64, 32, 64, 256), (3, 40, 8, 24, 64)])
def test_latent_with_expanded_keys(heads, dim, rot, vdim, rank):
    """Portions of which the long ones are expanded at the largest sizes (the cost rule keeps the others on the form that reads the latents), then one behind
    cached latents, and a step that mixes a long portion with a single token."""
    W = 64
    m = {"heads": heads, "dim": dim, "rot_dim": rot, "vdim": vdim, "kv_rank": rank, "q_rank": 48, "scale": (dim + rot) ** -0.5,
         "rot": {"dims": rot, "base": 10000.0, "scaling": {"factor": 4.0, "original": 256, "fast": 32.0, "slow": 1.0}}}
    cfg = {"architecture": "Fivedra", "vocab": 31, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5},
           "layers": [{"type": "latent_attention", "mixer": m, "mlp": None}]}
    w = FO.random_weights(cfg, heads)
    rows = inputs([1101, 600], W, 7)
    P = d64(w, "l0.mix.")
    wants = [FO.latent_attention(torch.from_numpy(r).double(), P, "", m, 1e-5).numpy() for r in rows]
    model = build(cfg, w, 16, {})
    check(model, rows, [[40, 600], [560, 0], [501, 0]], wants, W)
    check(model, rows, [[600, 0], [1, 599], [500, 1]], wants, W)
    model.close()


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("kind", ["grouped", "latent"])
def test_rows_that_do_not_see_a_value_stay_finite(kind, bad):
    """A token whose row holds a NaN or an infinity leaves the tokens before it as they are, also those that share its tile of keys or of rows."""
    W, at, n = 64, 437, 520
    if kind == "grouped":
        m = {"heads": 4, "kv_heads": 2, "dim": 64, "vdim": 64, "scale": 0.125}
        cfg = {"architecture": "Tutizen", "vocab": 31, "width": W, "norm": {"eps": 1e-5}, "residual_mult": 1.0, "layers": [{"type": "attention", "mixer": m, "mlp": None}]}
        w = TO.random_weights(cfg, 5)
        P = d64(w, "l0.mix.")
        want = lambda x: TO.attention(x, P, m, 1e-5)[0]           # noqa: E731
    else:
        m = {"heads": 20, "dim": 96, "rot_dim": 32, "vdim": 128, "kv_rank": 512, "q_rank": 48, "scale": 128 ** -0.5,
             "rot": {"dims": 32, "base": 10000.0, "scaling": {"factor": 4.0, "original": 256, "fast": 32.0, "slow": 1.0}}}
        cfg = {"architecture": "Fivedra", "vocab": 31, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5},
               "layers": [{"type": "latent_attention", "mixer": m, "mlp": None}]}
        w = FO.random_weights(cfg, 6)
        P = d64(w, "l0.mix.")
        want = lambda x: FO.latent_attention(x, P, "", m, 1e-5)   # noqa: E731
    row = inputs([n], W, 11)[0]
    ref = want(torch.from_numpy(row).double()).numpy()
    row[at, 5] = bad
    model = build(cfg, w, 16, {})
    got = model.engine.run_part(0, 2, [model.admit()], [n], row)
    model.close()
    assert np.isfinite(got[:at]).all() and not np.isfinite(got[at:]).all(-1).any()
    err = np.sqrt(((got[:at] - ref[:at]) ** 2).mean(-1)) / np.sqrt((ref[:at] ** 2).mean(-1))
    assert err.max() < TOL


def latent_groups(model, behind, count):
    """The launch groups of a step of `count` tokens behind `behind` cached positions."""
    s = model.admit()
    model.engine.set_length(s, behind)
    out = set(model.engine.profile_step([s], [count], 1))
    model.release(s)
    return out


def test_the_latent_choice_counts_the_keys_under_the_window():
    """A short portion behind a long context expands the latents where it sees all of them and reads them as they are where a window hides most."""
    import test_gpu_karusun as K
    for window, expands in ((100000, True), (512, False)):
        cfg = K.config([K.lat(heads=20, dim=96, rot_dim=32, vdim=128, kv_rank=512, window=window)], width=64, vocab=40, groups=1, taps=2)
        model = K.build(cfg, K.make_weights(cfg, 3), "bfloat16", max_tokens=4096, page_size=16, max_step_tokens=1024)
        assert ("latent.expand_gemm" in latent_groups(model, 3000, 64)) == expands
        assert "latent.expand_gemm" in latent_groups(model, 0, 1000)
        model.close()


@pytest.mark.parametrize("heads,dim,rot,vdim,rank", [(8, 64, 32, 64, 256), (3, 40, 8, 24, 64), (5, 24, 0, 128, 80), (7, 120, 8, 8, 32)])
def test_latent_form_with_expanded_keys_at_small_sizes(heads, dim, rot, vdim, rank, monkeypatch):
    """The same where its cost rule would decide otherwise: odd head counts, heads below a swizzle block, sequences whose rows start between tiles."""
    monkeypatch.setenv("WF_SEQ_ATTN_MMA", "4")
    W = 64
    m = {"heads": heads, "dim": dim, "rot_dim": rot, "vdim": vdim, "kv_rank": rank, "q_rank": 48, "scale": (dim + rot) ** -0.5,
         "rot": {"dims": rot, "base": 10000.0, "scaling": {"factor": 4.0, "original": 256, "fast": 32.0, "slow": 1.0}}}
    cfg = {"architecture": "Fivedra", "vocab": 31, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5},
           "layers": [{"type": "latent_attention", "mixer": m, "mlp": None}]}
    w = FO.random_weights(cfg, heads)
    lens = [333, 70, 190]
    rows = inputs(lens, W, 7)
    P = d64(w, "l0.mix.")
    wants = [FO.latent_attention(torch.from_numpy(r).double(), P, "", m, 1e-5).numpy() for r in rows]
    model = build(cfg, w, 16, {})
    assert "latent.expand_gemm" in latent_groups(model, 0, 40)
    check(model, rows, [[200, 3, 129], [5, 66, 0], [128, 1, 61]], wants, W)
    model.close()


def test_latent_sizes_without_a_tensor_core_form_keep_the_plain_kernel(monkeypatch):
    """Ranks that no mma.sync form takes had float queries and weights: asked for or not, they are not expanded."""
    monkeypatch.setenv("WF_SEQ_ATTN_MMA", "4")
    m = {"heads": 20, "dim": 96, "rot_dim": 32, "vdim": 128, "kv_rank": 504, "q_rank": 48, "scale": 128 ** -0.5, "rot": {"dims": 32, "base": 10000.0}}
    cfg = {"architecture": "Fivedra", "vocab": 31, "width": 64, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5},
           "layers": [{"type": "latent_attention", "mixer": m, "mlp": None}]}
    model = build(cfg, FO.random_weights(cfg, 2), 16, {})
    assert "latent.expand_gemm" not in latent_groups(model, 0, 600)
    model.close()


@pytest.mark.parametrize("window", [1, 130, 300])
def test_windowed_latent_form_with_expanded_keys(window, monkeypatch):
    import test_gpu_karusun as K
    monkeypatch.setenv("WF_SEQ_ATTN_MMA", "4")
    cfg = K.config([K.lat(heads=5, dim=40, rot_dim=16, vdim=24, kv_rank=80, window=window)], width=64, vocab=40, groups=1, taps=2)
    w = K.make_weights(cfg, 8)
    model = K.build(cfg, w, "bfloat16", max_tokens=1024, page_size=16, max_step_tokens=512)
    assert "latent.expand_gemm" in latent_groups(model, 0, 40)
    x = inputs([500], 64, 9)[0]
    P = {k: torch.from_numpy(v).double() for k, v in K.O.sub(w, "l0.mix.").items()}
    want = K.O.latent_attention(torch.from_numpy(x).double(), P, cfg["layers"][0]["mixer"], 1e-6).numpy()
    check(model, [x], [[260], [3], [237]], [want], 64)
    model.close()
